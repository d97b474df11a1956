"""Grid reductions against math.fsum (exactly rounded sums): the WRMS norm's groups of four terms
and its reciprocal, the block-wide sum of the partials, the CFL speed.  A norm's terms each carry
a few roundings (2^-53 relative), which a sum of positive terms keeps, so 1e-14 relative bounds
every size; totals are compensated: 1e-15."""
import math

import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu


# cells x fields below and above one group of four per thread (262144 threads), odd remainders
@pytest.mark.parametrize("shape,nchem", [((3, 3, 3), 0), ((17, 13, 11), 2), ((64, 64, 65), 0),
                                         ((70, 61, 67), 10), ((128, 96, 90), 0)])
def test_reductions_match_exact_sums(cuda, shape, nchem):
    torch = cuda
    import gbmv
    rng = np.random.default_rng(5)
    wl = W.rayleigh_taylor(shape=shape, nchem=nchem, seed=W.SEED_BASE + 710)
    w = wl["fields"]
    v = [1e-6 * rng.standard_normal(f.shape) for f in w]
    h = gbmv.Hydro(shape, nchem, wl["bc"], wl["gamma"], None)
    wt = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in w]
    vt = [torch.from_numpy(f).cuda() for f in v]
    q = np.concatenate([(a / (1e-6 * np.abs(b) + 1e-11)).ravel() for a, b in zip(v, w)])
    ref = math.sqrt(math.fsum(q * q) / q.size)
    assert abs(h.wrms_norm(vt, wt, 1e-6, 1e-11) - ref) <= 1e-14 * ref
    m, e = h.check_conservation(wt)
    for got, f in ((m, w[0]), (e, w[4])):
        exact = math.fsum(f.ravel())
        assert abs(got - exact) <= 1e-15 * abs(exact)
    p = (wl["gamma"] - 1) * (w[4] - 0.5 * (w[1] ** 2 + w[2] ** 2 + w[3] ** 2) / w[0])
    a = np.max(np.abs(w[1] / w[0]) + np.sqrt(wl["gamma"] * p / w[0]))
    dt = 0.5 * min(1.0 / n for n in shape) / a
    assert abs(h.stability(wt, 0.5) - dt) <= 1e-14 * dt


def test_wrms_norm_extreme_weights(cuda):
    """Weights outside the range of the fast reciprocal: tiny and huge |y|, a zero denominator."""
    torch = cuda
    import gbmv
    shape = (5, 4, 3)
    h = gbmv.Hydro(shape, 0, (0,) * 6, 1.4, None)
    for y, v in ((1e-312, 1e-312), (1e305, 1e300), (1e-300, 1e-303)):
        yt = [torch.full((3, 4, 5), y, dtype=torch.float64, device="cuda") for _ in range(5)]
        vt = [torch.full((3, 4, 5), v, dtype=torch.float64, device="cuda") for _ in range(5)]
        got = h.wrms_norm(vt, yt, 1.0, 0.0)
        if y < 1e-309:  # the weight 1 / y itself is not a double
            assert not math.isfinite(got)
        else:
            ref = v * (1.0 / y)
            assert abs(got - ref) <= 1e-9 * ref
    zt = [torch.zeros((3, 4, 5), dtype=torch.float64, device="cuda") for _ in range(5)]
    # a zero denominator gives an infinite term; the compensated accumulation turns it into NaN
    assert not math.isfinite(h.wrms_norm(vt, zt, 1.0, 0.0))
