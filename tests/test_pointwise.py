"""Routines that reach the reference's bits another way, against the oracle
(the product against IEEE arithmetic): the integer-pipe product, the bisection that evaluates the cubic only where rounding can hide its sign,
and the cube root from a single-precision start.  Equality is exact."""

import numpy as np
import pytest

from swe_fvm_gb300 import _lib

N = 40000


def run(kind, args, device):
    a = np.ascontiguousarray(args, dtype=np.float64)
    out = np.empty(a.shape[0])
    st = _lib.load().swe_selftest_pointwise(kind, a.shape[0], a.ctypes.data, out.ctypes.data, int(device))
    assert st == 0
    return out


def one_vertex_dry(rng, n):
    """PartWet2's cubic on [0, 1]: c = (alpha - 3) / beta, d = (1 + beta - alpha) / beta^2."""
    alpha, beta = 3.0 * rng.random(n), 10.0 ** (-6 * rng.random(n) ** 3)
    z = np.zeros(n)
    return np.stack([(1 + beta - alpha) / (beta * beta), (alpha - 3) / beta, z, z, z + 1.0], 1)


def partly_wet_level(rng, n):
    """PartWet1's cubic on [b12, b13], from steep cells to nearly flat ones on a high bed, and beds below zero."""
    z = rng.random((n, 3))
    flat = rng.random(n) < 0.5
    z[flat, 1:] = z[flat, :1] + 10.0 ** rng.uniform(-7, -1, (flat.sum(), 1)) * rng.random((flat.sum(), 2))
    z -= np.where(rng.random(n) < 0.3, 0.5, 0.0)[:, None]
    b13, b23, bc = z.max(1), z.min(1), z.mean(1)
    b12 = 3 * bc - b23 - b13
    w = b12 + (b13 - b12) * rng.random(n)
    h = w - bc
    c = 3 * (b12 * b13 + b13 * b23 - b12 * b23)
    d = (b13 - b23) * (3 * h * (b13 - b12) - b12 * (b12 + b23)) - b23 * b23 * b13
    return np.stack([d, c, -3 * b13, b12, b13], 1)[b13 > b12]


def any_cubic(rng, n):
    """Any coefficients and interval, several roots, roots on the ends and on dyadic points among them."""
    s = lambda: rng.standard_normal(n) * 10.0 ** (2 * rng.standard_normal(n))  # noqa: E731
    x0, c, b = s(), s(), s()
    x1 = x0 + np.abs(s()) + 1e-9
    r = x0 + (x1 - x0) * rng.choice([0.0, 1.0, 0.5, 0.25, 0.3], n)
    d = np.where(rng.random(n) < 0.5, s(), -(r * r * r + b * r * r + c * r))
    unit = rng.random(n) < 0.4
    x0, x1, b = np.where(unit, 0.0, x0), np.where(unit, 1.0, x1), np.where(unit, 0.0, b)
    d = np.where(unit & (rng.random(n) < 0.1), rng.choice([0.0, -0.0, 1e-300, -1e-20], n), d)
    return np.stack([d, c, b, x0, x1], 1)


def check_bisection(make, device):
    from oracle import oracle

    L = oracle.lib()
    a = make(np.random.default_rng(11), N)
    got = run(0, a, device)
    want = np.array([L.oracle_bisection_cubic(*row) for row in a])
    assert np.array_equal(got.view(np.int64), want.view(np.int64))


def check_cbrt(device):
    from oracle import oracle

    L = oracle.lib()
    rng = np.random.default_rng(12)
    whole = np.floor(rng.random(2000) * 1e5)
    x = np.concatenate([rng.standard_normal(N) * np.exp(100 * rng.standard_normal(N)), rng.random(N) ** 9,
                        whole ** 3, rng.random(100) * 1e-310, [0.0, -0.0, np.inf, -np.inf, 5e-324, 1.7e308]])
    got = run(1, x[:, None], device)
    want = np.array([L.oracle_cbrt_rn(v) for v in x])
    assert np.array_equal(got.view(np.int64), want.view(np.int64))


def operands(rng, n):
    """Products over exponents of every range, ties, powers of two, zeros, subnormals and specials."""
    def one():
        exp = np.where(rng.random(n) < 0.6, rng.integers(1003, 1043, n),
                       np.where(rng.random(n) < 0.5, rng.integers(505, 1540, n), rng.integers(0, 2048, n)))
        man = rng.integers(0, 1 << 52, n)
        man = np.where(rng.random(n) < 0.3, man & ~((1 << 27) - 1), man)  # short ones: exact products and ties
        man = np.where(rng.random(n) < 0.1, rng.choice([0, 1, (1 << 52) - 1, 1 << 51], n), man)
        x = ((rng.integers(0, 2, n) << 63) | (exp << 52) | man).astype(np.int64).view(np.float64)
        return np.where(rng.random(n) < 0.05, rng.choice([0.0, -0.0, np.inf, np.nan, 5e-324, 1.0], n), x)

    return np.stack([one(), one()], 1)


@pytest.mark.gpu
def test_product_device(gpu):
    """The integer product has the FP64 instruction's bits, or says that it leaves the operands to it: never for
    zeros and exponents from 2^-510 to 2^510."""
    a = operands(np.random.default_rng(13), 400000)
    got = run(2, a, True).view(np.int64)
    with np.errstate(all="ignore"):
        want = (a[:, 0] * a[:, 1]).view(np.int64)
    left = got == 0x7FF8000000000123
    assert np.array_equal(got[~left], want[~left])
    mag = np.abs(a)
    fine = ((mag == 0) | ((mag > 2.0 ** -510) & (mag < 2.0 ** 510))).all(1)
    assert not (left & fine).any()
    assert fine.sum() > 100000 and left.sum() > 10000


MAKES = [one_vertex_dry, partly_wet_level, any_cubic]


@pytest.mark.parametrize("make", MAKES)
def test_bisection_host(make):
    check_bisection(make, False)


def test_cbrt_host():
    check_cbrt(False)


@pytest.mark.gpu
@pytest.mark.parametrize("make", MAKES)
def test_bisection_device(gpu, make):
    check_bisection(make, True)


@pytest.mark.gpu
def test_cbrt_device(gpu):
    check_cbrt(True)
