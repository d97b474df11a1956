"""The float-float reconstructions between the sizes at which their arithmetic changes, against the
oracle: linear ramps whose jumps per cell cross the point where the weights are scaled.  The states
keep velocities and sound speeds near 1, so the mixed form's parity bar is 1e-9 of the largest
tendency (its roundings are 2^-46, times the flux over its difference, ~100 here); the FP64 form's
own error is held to 1e-11, so that a broken reference could not pass."""
import numpy as np
import pytest

import oracle_py as O
from conftest import maxnorm_err

pytestmark = pytest.mark.gpu

GAMMA = 1.4


def _ramp_state(shape, nchem, lo, hi, fluid):
    """Rows along x with slopes from lo to hi, a per cent or two apart: of the density at constant
    temperature (fluid), or of every tracer in a uniform gas."""
    nx, ny, nz = shape
    slope = np.geomspace(lo, hi, ny * nz).reshape(nz, ny, 1)
    ramp = slope * (1.0 + np.arange(nx))
    rho = ramp.copy() if fluid else np.ones((nz, ny, nx))
    u = (0.5, 0.25, -0.375)
    p = rho.copy()
    f = [rho] + [rho * x for x in u]
    f.append(p / (GAMMA - 1.0) + 0.5 * rho * sum(x * x for x in u))
    if nchem:
        f.append(np.repeat((rho if fluid else ramp)[..., None], nchem, axis=3))
    return f


def _check(torch, shape, nchem, bc, fields, tol, precisions):
    import gbmv
    st, ref = O.feuler(fields, nchem, bc, GAMMA, None)
    assert st == 0
    w = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in fields]
    h = gbmv.Hydro(shape, nchem, bc, GAMMA, None)
    for precision in (gbmv.FP64,) + precisions:
        out = [torch.full_like(f, np.nan) for f in w]
        assert h.fEuler(0.0, w, out, precision) == 0
        for v, (a, r) in enumerate(zip(out, ref)):
            a = a.cpu().numpy()
            assert np.isfinite(a).all(), (precision, v)
            bar = 1e-11 if precision == gbmv.FP64 else tol
            if precision == gbmv.MIXED_FAST and v == 5:
                bar = 1e-6
            assert maxnorm_err(a, r) <= bar, (precision, v)


@pytest.mark.parametrize("lo,hi", [(1e-2, 1.0), (1.0, 100.0), (100.0, 1e4)])
@pytest.mark.parametrize("fluid", [False, True])
def test_ramps_across_the_scaling_of_the_weights(cuda, fluid, lo, hi):
    import gbmv
    shape, bc = (12, 30, 20), (1, 1, 0, 0, 1, 1)
    fields = _ramp_state(shape, 2, lo, hi, fluid)
    _check(cuda, shape, 2, bc, fields, 1e-9, (gbmv.MIXED, gbmv.MIXED_FAST))
