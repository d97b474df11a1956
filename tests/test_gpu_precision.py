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
