"""The float-float reconstructions between the sizes at which their arithmetic changes, against the
oracle: linear ramps whose jumps per cell cross the point where the weights are scaled, and tracers
at both ends of the float range.  The ramps keep velocities and sound speeds near 1, so the mixed
form's parity bar is 1e-9 of the largest tendency (its roundings are 2^-46, times the flux over its
difference, ~100 here); the FP64 form's own error is held to 1e-11, so that a broken reference could
not pass."""
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


def _tracer_state(shape, nchem, size, seed):
    """Uniform density and pressure, velocities of a few tenths, tracers of the given size."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = shape
    rho = np.ones((nz, ny, nx))
    u = rng.uniform(-0.3, 0.3, (3, nz, ny, nx))
    f = [rho, u[0], u[1], u[2], 1.0 / (GAMMA - 1.0) + 0.5 * (u * u).sum(0)]
    f.append(size * rng.uniform(0.5, 1.5, (nz, ny, nx, nchem)))
    return f


# fluxes whose float pairs reach the end of the float range, where the pairs themselves lose bits
# (2^-149 absolute: a few dozen such roundings make a tendency); FP32 weights keep the contract's 1e-6
@pytest.mark.parametrize("size", [1e-18, 1e-24, 1e-28, 1e-30, 1e-32, 1e-34, 1e-36])
def test_small_tracers(cuda, size):
    import gbmv
    shape, bc = (17, 12, 9), (3, 3, 0, 0, 1, 1)
    fields = _tracer_state(shape, 2, size, 7)
    _check(cuda, shape, 2, bc, fields, 1e-12 + 64 * 2.0 ** -149 / size, (gbmv.MIXED,
                                                                        gbmv.MIXED_FAST))


# on both sides of the FP64 fallback (fluxes of 1e18, 1e15 scaled) up to the end of the float range
@pytest.mark.parametrize("size", [1e12, 7e14, 2e15, 1e16, 1e17, 3e18, 1e20, 1e30, 5e36])
def test_large_tracers(cuda, size):
    import gbmv
    shape, bc = (5, 4, 3), (3, 3, 0, 0, 1, 1)
    fields = _tracer_state(shape, 2, size, 8)
    _check(cuda, shape, 2, bc, fields, 1e-12, (gbmv.MIXED, gbmv.MIXED_FAST))


def test_fluid_errors_beside_fp64(cuda):
    """The fluid tendencies' largest errors in units of the FP64 form's, averaged over fields and
    velocity scales: normalised float-float operations (2^-47 beside 2^-53, errors partly averaged
    out) measured 24.0, sums of products left un-normalised in the projections 28.7."""
    torch = cuda
    import gbmv
    import workloads as W
    shape, ratios = (24, 20, 16), []
    for v, rho in ((1.0, 1.0), (30.0, 40.0), (1e3, 1.0), (1e4, 1e2), (1e5, 1.0), (1e6, 1.0)):
        worst = np.zeros((2, 5))
        for seed in range(6):
            wl = W.rayleigh_taylor(shape=shape, nchem=0, seed=W.SEED_BASE + 7000 + seed)
            f = wl["fields"]
            f = [f[0] * rho, f[1] * rho * v, f[2] * rho * v, f[3] * rho * v, f[4] * rho * v * v]
            st, ref = O.feuler(f, 0, wl["bc"], wl["gamma"], None)
            assert st == 0
            w = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in f]
            h = gbmv.Hydro(shape, 0, wl["bc"], wl["gamma"], None)
            for precision in (gbmv.FP64, gbmv.MIXED):
                out = [torch.full_like(x, np.nan) for x in w]
                assert h.fEuler(0.0, w, out, precision) == 0
                e = [maxnorm_err(a.cpu().numpy(), r) for a, r in zip(out, ref)]
                worst[precision] = np.maximum(worst[precision], e)
        assert worst[0].max() <= 1e-7  # eps times the basis' condition ~ v at sound speeds ~ v
        ratios.append(worst[1] / worst[0])
    assert np.mean(ratios) <= 26.0
