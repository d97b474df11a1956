"""Precision kept where fewer FP64 instructions took a literal formula's place."""
from decimal import Decimal, getcontext
from fractions import Fraction
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one large and three small squares, a quarter of the 128 x 128 x 64 grid apart, which is where one
# thread's next terms lie: a plain sum of the four is 1.26 units in the last place of the norm away
# for these values, a compensated one 0.27 (the rounding of the quotient and of the root)
@pytest.mark.parametrize("big,small", [("0x1.04c050b30a648p+0", "0x1.6a0f7efd9260dp-27"),
                                       ("0x1.048013f9651b6p+0", "0x1.6a17a82985975p-27"),
                                       ("0x1.0467ba0374572p+0", "0x1.6a74b8550b199p-27")])
def test_wrms_terms_are_compensated(cuda, big, small):
    torch = cuda
    import gbmv
    big, small = float.fromhex(big), float.fromhex(small)
    shape = (128, 128, 64)
    h = gbmv.Hydro(shape, 0, (0,) * 6, 1.4, None)
    n = shape[0] * shape[1] * shape[2]
    v = torch.full((n,), small, dtype=torch.float64, device="cuda")
    v[:n // 4] = big
    v = v.view(64, 128, 128)
    y = torch.zeros_like(v)
    got = h.wrms_norm([v] * 5, [y] * 5, 1e-6, 1.0)  # unit weights
    getcontext().prec = 50
    mean = (Fraction(big) ** 2 + 3 * Fraction(small) ** 2) / 4
    exact = (Decimal(mean.numerator) / Decimal(mean.denominator)).sqrt()
    assert abs(Decimal(got) - exact) <= Decimal(math.ulp(got)) * Decimal("0.75")


@pytest.mark.parametrize("rho_vacuum", [1.2e-308, 1e-310])
def test_derivatives_beside_a_subnormal_density(cuda, rho_vacuum):
    """A near-vacuum cell whose density is below the range of the approximate reciprocal (the first's
    reciprocal is a double still): the products elsewhere are those beside one of 1e-290 (both
    vanish beside the neighbours' numbers; 1e-10 leaves their roundings a wide margin)."""
    torch = cuda
    import gbmv
    shape, bc = (9, 8, 7), (0, 0, 1, 1, 3, 3)
    rng = np.random.default_rng(3)
    n = (shape[2], shape[1], shape[0])
    w0 = [rng.uniform(0.5, 1.5, n)] + [rng.uniform(-0.2, 0.2, n) for _ in range(3)]
    w0.append(rng.uniform(2.0, 3.0, n))
    d0, v0 = ([rng.standard_normal(n) for _ in range(5)] for _ in range(2))
    at = (3, 4, 4)
    other = np.ones(n, dtype=bool)
    other[at] = False
    h = gbmv.Hydro(shape, 0, bc, 1.4, None)
    out = []
    for rho in (rho_vacuum, 1e-290):
        for f, x in zip(w0, (rho, 0.0, 0.0, 0.0, 2.5 * rho)):
            f[at] = x
        for f in d0:
            f[at] = 0.0
        w, dw, v = ([torch.from_numpy(f).cuda() for f in g] for g in (w0, d0, v0))
        jv, vj = ([torch.full_like(f, np.nan) for f in w] for _ in range(2))
        assert h.fEuler_jvp(0.0, w, dw, jv) == 0
        assert h.fEuler_vjp(0.0, w, v, vj) == 0
        out.append([x.cpu().numpy() for x in jv + vj])
    for k, (a, b) in enumerate(zip(*out)):
        a, b = a[other], b[other]
        assert np.isfinite(b).all(), k
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b)), k


def test_wave_speed_at_a_tiny_density(cuda):
    """A density whose reciprocal is not a double: the speed is that of the quotients."""
    torch = cuda
    import gbmv
    shape = (4, 3, 3)
    h = gbmv.Hydro(shape, 0, (0,) * 6, 1.4, None)
    w = [torch.full((3, 3, 4), x, dtype=torch.float64, device="cuda")
         for x in (1e-310, 5e-311, 0.0, 0.0, 1e-310)]
    alpha = 0.5 + math.sqrt(1.4 * 0.4)
    dt = 0.5 * 0.25 / alpha
    assert abs(h.stability(w, 0.5) - dt) <= 1e-12 * dt


def _ulps(got, exact):
    """Error of the doubles got against extended-precision numbers, in units in the last place."""
    ulp = np.spacing(np.abs(exact).astype(np.float64)).astype(np.longdouble)
    return np.abs((got.astype(np.longdouble) - exact) / ulp)


def _functions(torch, tables, x):
    import gbmv
    c = gbmv.Chem(1, tables)
    return gbmv.diag_math(c, torch.from_numpy(x).cuda()).cpu().numpy()


def _doubles(rng, n, lo, hi):
    """Doubles of either sign, exponents lo .. hi - 1: random, and the ends of a binade."""
    m = 1.0 + rng.integers(0, 1 << 52, n) * 2.0 ** -52
    m[:n // 8] = 1.0
    m[n // 8:n // 4] = 2.0 - 2.0 ** -52
    return np.ldexp(m, rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)


# r (1 + e + e^2) with |e| < 2^-20: half a unit for the last rounding, 2^-60 for e^3
def test_reciprocals(cuda, tables):
    rng = np.random.default_rng(1)
    one = np.longdouble(1)
    x = _doubles(rng, 1 << 19, -1021, 1021)
    r, _, q, _ = _functions(cuda, tables, x)
    assert _ulps(r, one / x).max() <= 0.51
    assert _ulps(q, 3 * one / x).max() <= 1.6  # 3 r: the reciprocal's rounding and the product's
    x = _doubles(rng, 1 << 19, -1000, 1000)
    assert _ulps(_functions(cuda, tables, x)[1], 2 * one / x).max() <= 0.51
    # outside the approximate instruction's range: the division, bit for bit
    x = np.concatenate([_doubles(rng, 4096, -1074, -1021), _doubles(rng, 4096, 1021, 1024),
                        [5e-324, -5e-324, 0.0, -0.0, np.inf, -np.inf, np.nan]])
    r, _, q, _ = _functions(cuda, tables, x)
    with np.errstate(divide="ignore", over="ignore"):
        ok = np.abs(x) != np.ldexp(1.0, -1021)
        assert np.array_equal(r[ok], (1.0 / x)[ok], equal_nan=True)
        assert np.array_equal(q[ok], (3.0 / x)[ok], equal_nan=True)


def test_temperature_logarithm(cuda, tables):
    """Six terms of the series leave 2^-58 absolute; the table's entry carries more bits than a
    double, so the last addition's rounding is the only other error."""
    rng = np.random.default_rng(2)
    inside = np.exp2(rng.uniform(-2.0, 18.0, 1 << 19))
    edges = np.ldexp(1.0 + np.arange(129) / 128.0, 0)[None] * np.exp2(np.arange(-2, 17))[:, None]
    edges = np.concatenate([edges.ravel(), np.nextafter(edges, 0).ravel()])
    x = np.concatenate([inside, edges[(edges >= 0.25) & (edges < 2.0 ** 18)]])
    exact = np.log(x.astype(np.longdouble))
    got = _functions(cuda, tables, x)[3]
    half = 0.5 * np.spacing(np.abs(exact).astype(np.float64))
    assert np.all(np.abs(got - exact) <= 1.01 * half + 2.0 ** -57.5)
    x = np.concatenate([np.exp2(rng.uniform(-40, -2.01, 4096)), np.exp2(rng.uniform(18.0, 60, 4096))])
    assert _ulps(_functions(cuda, tables, x)[3], np.log(x.astype(np.longdouble))).max() <= 1.0
