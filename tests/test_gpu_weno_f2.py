"""The float-float sweeps over the range of magnitudes their reconstructions split on: small jumps
(weights as they are), jumps beyond ~1000 (weights scaled by a power of two), states whose faces
leave the float range (FP64 per face), and each register budget.  Against the oracle.  Tolerances:
the projections' condition grows with the sound speed (the basis holds c^2 where c is expected) and
the fluxes cancel, so each field's bound is the FP64 form's own error on the same state, by the ratio
of the roundings -- float-float results keep 46 bits or more, 2^7 of FP64's -- and a factor two, or
1e-9 where that is larger; GBMV_MIXED_FAST the same for the fluid, 1e-6 for the tracers."""
import numpy as np
import pytest

import oracle_py as O
import workloads as W
from conftest import maxnorm_err

pytestmark = pytest.mark.gpu


def _state(shape, nchem, v, rho, seed):
    """The Rayleigh-Taylor state in other units: densities times rho, velocities times v."""
    wl = W.rayleigh_taylor(shape=shape, nchem=nchem, seed=seed)
    f = wl["fields"]
    out = [f[0] * rho, f[1] * rho * v, f[2] * rho * v, f[3] * rho * v, f[4] * rho * v * v]
    if nchem:
        out.append(f[5] * rho)
    return out, wl["gamma"]


@pytest.mark.parametrize("v,rho", [(1.0, 1.0), (1e-4, 1e-3), (30.0, 40.0), (1e3, 1e2), (1e4, 1e5),
                                   (1e6, 1e4)])
@pytest.mark.parametrize("nchem", [0, 6])
@pytest.mark.parametrize("shape", [(3, 3, 3), (17, 12, 9)])
def test_f2_sweeps_over_magnitudes(cuda, v, rho, nchem, shape):
    torch = cuda
    import gbmv
    bc = (3, 3, 0, 0, 1, 3)
    fields, gamma = _state(shape, nchem, v, rho, W.SEED_BASE + 720)
    st, ref = O.feuler(fields, nchem, bc, gamma, None)
    assert st == 0
    w = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in fields]
    out = [torch.full_like(f, np.nan) for f in w]
    assert gbmv.Hydro(shape, nchem, bc, gamma, None).fEuler(0.0, w, out, gbmv.FP64) == 0
    tol = [max(1e-9, 256 * maxnorm_err(a.cpu().numpy(), r)) for a, r in zip(out, ref)]
    for precision in (gbmv.MIXED, gbmv.MIXED_FAST):
        if precision == gbmv.MIXED_FAST and nchem:
            tol[5] = 1e-6
        first = None
        for shared in (False, True):
            h = gbmv.Hydro(shape, nchem, bc, gamma, None)
            h.set_sweep_budget(shared)
            out = [torch.full_like(f, np.nan) for f in w]
            assert h.fEuler(0.0, w, out, precision) == 0
            for a, r, t in zip(out, ref, tol):
                assert maxnorm_err(a.cpu().numpy(), r) <= t, (precision, shared)
            if first is None:
                first = out
            assert all(torch.equal(a, b) for a, b in zip(out, first))


def test_f2_sweeps_forcing_and_dirichlet(cuda):
    """A forcing already in wdot, and homogeneous Dirichlet faces (negated densities: FP64 faces,
    NaN where the reference has NaN)."""
    torch = cuda
    import gbmv
    shape, bc = (9, 8, 7), (2, 2, 0, 0, 3, 1)
    fields, gamma = _state(shape, 4, 1.0, 1.0, W.SEED_BASE + 721)
    _, ref = O.feuler(fields, 4, bc, gamma, None)
    w = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in fields]
    h = gbmv.Hydro(shape, 4, bc, gamma, None)
    for precision, tol in ((gbmv.MIXED, 1e-9), (gbmv.MIXED_FAST, 1e-6)):
        out = [torch.full_like(f, 0.5) for f in w]
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        h.fEuler_async(0.0, w, out, status, precision, gbmv.FORCE_IN_WDOT)
        for a, r in zip(out, ref):
            assert maxnorm_err(a.cpu().numpy(), r + 0.5) <= tol
