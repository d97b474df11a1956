"""The FP64 flux divergence's launch forms against the oracle: two threads a face on small grids,
one on larger ones (both sides of the line, and face counts that leave a partial warp), the
primitives from the cell pass or formed per stencil point (a forcing already in wdot, an in-place
call).  Tolerance: the FP64 parity bar, 1e-12 of each field's largest magnitude; the largest
difference expected is ~1e-13 (a few roundings of a flux, divided by the spacing)."""
import numpy as np
import pytest

import oracle_py as O
import workloads as W
from conftest import maxnorm_err

pytestmark = pytest.mark.gpu

# 9728 faces is the line: (16, 16, 11) has 9056, (16, 16, 12) 9856; the others leave odd remainders
SHAPES = [(3, 3, 3), (7, 5, 3), (16, 16, 11), (16, 16, 12), (33, 17, 21)]
BCS = [(0, 0, 0, 0, 0, 0), (3, 3, 1, 3, 0, 0)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("nchem", [0, 10])
@pytest.mark.parametrize("bc", BCS)
def test_fp64_forms_match_oracle(cuda, shape, nchem, bc):
    torch = cuda
    import gbmv
    wl = W.rayleigh_taylor(shape=shape, nchem=nchem, seed=W.SEED_BASE + 700)
    st, ref = O.feuler(wl["fields"], nchem, bc, wl["gamma"], None)
    assert st == 0
    h = gbmv.Hydro(shape, nchem, bc, wl["gamma"], None)
    w = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in wl["fields"]]
    plain = [torch.full_like(f, np.nan) for f in w]
    assert h.fEuler(0.0, w, plain) == 0
    forced = [torch.full_like(f, 0.25) for f in w]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    h.fEuler_async(0.0, w, forced, status, gbmv.FP64, gbmv.FORCE_IN_WDOT)
    inplace = [f.clone() for f in w]
    assert h.fEuler(0.0, inplace, inplace) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for a, b, c, r in zip(plain, forced, inplace, ref):
        assert maxnorm_err(a.cpu().numpy(), r) <= 1e-12
        assert maxnorm_err(b.cpu().numpy(), r + 0.25) <= 1e-12
        assert maxnorm_err(c.cpu().numpy(), r) <= 1e-12


def test_fp64_forms_flag_illegal_states(cuda):
    torch = cuda
    import gbmv
    wl = W.rayleigh_taylor(shape=(9, 8, 7), nchem=2, seed=W.SEED_BASE + 701)
    h = gbmv.Hydro((9, 8, 7), 2, wl["bc"], wl["gamma"], None)
    for field, bit in ((0, 1), (4, 2)):
        bad = [f.copy() for f in wl["fields"]]
        bad[field][3, 2, 1] = -1.0
        w = [torch.from_numpy(f).cuda() for f in bad]
        for flags in (0, gbmv.FORCE_IN_WDOT):
            out = [torch.zeros_like(f) for f in w]
            status = torch.zeros(1, dtype=torch.int32, device="cuda")
            h.fEuler_async(0.0, w, out, status, gbmv.FP64, flags)
            assert int(status.item()) & bit


@pytest.mark.parametrize("nchem", [0, 4])
def test_jvp_in_place_matches_out_of_place(cuda, nchem):
    """jv may be dw itself: the primitives are then formed per stencil point instead of in jv.
    The two forms differ by the rounding of the velocities and the pressure (~1e-15 per flux)."""
    torch = cuda
    import gbmv
    wl = W.rayleigh_taylor(shape=(13, 9, 7), nchem=nchem, seed=W.SEED_BASE + 702)
    h = gbmv.Hydro((13, 9, 7), nchem, (3, 3, 0, 0, 1, 3), wl["gamma"], None)
    w = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in wl["fields"]]
    gen = torch.Generator(device="cuda").manual_seed(3)
    d = [torch.rand(f.shape, generator=gen, device="cuda", dtype=torch.float64) - 0.5 for f in w]
    out = [torch.empty_like(f) for f in w]
    h.fEuler_jvp(0.0, w, d, out)
    h.fEuler_jvp(0.0, w, d, d)
    for a, b in zip(d, out):
        assert maxnorm_err(a.cpu().numpy(), b.cpu().numpy()) <= 1e-12


def test_fp64_sweeps_at_large_densities(cuda):
    """Flux jumps beyond 2^112 take the scaled weights.  The equations are homogeneous of degree one
    in the conserved fields and the tracers, and so is the scheme where the weights' 1e-6 is
    negligible: from densities in 2^60 to 2^200 the right-hand side scales, the derivatives stay.
    All factors are powers of two, so only the roundings of the scaled weights differ: 1e-12."""
    torch = cuda
    import gbmv
    shape, nchem = (11, 9, 7), 4
    wl = W.rayleigh_taylor(shape=shape, nchem=nchem, seed=W.SEED_BASE + 703)
    h = gbmv.Hydro(shape, nchem, (3, 3, 0, 0, 1, 3), wl["gamma"], None)
    gen = torch.Generator(device="cuda").manual_seed(4)
    v = [torch.rand(f.shape, generator=gen, device="cuda", dtype=torch.float64) - 0.5
         for f in wl["fields"]]
    res = []
    for lam in (2.0 ** 60, 2.0 ** 200):
        w = [lam * torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in wl["fields"]]
        f, jv, u = ([torch.empty_like(x) for x in w] for _ in range(3))
        assert h.fEuler(0.0, w, f) == 0
        h.fEuler_jvp(0.0, w, v, jv)
        h.fEuler_vjp(0.0, w, v, u)
        _, ref = O.feuler([x.cpu().numpy() for x in w], nchem, (3, 3, 0, 0, 1, 3), wl["gamma"], None)
        for a, r in zip(f, ref):
            assert maxnorm_err(a.cpu().numpy(), r) <= 1e-12
        res.append([x.cpu().numpy() / lam for x in f] + [x.cpu().numpy() for x in jv + u])
    for a, b in zip(*res):
        assert maxnorm_err(a, b) <= 1e-12


# 4864 faces is the line between four threads a face and two: (11, 11, 12) has 4741 faces, (12, 11,
# 12) 5160; the Sod tube's grid; odd face counts in every direction
@pytest.mark.parametrize("shape", [(128, 3, 3), (11, 11, 12), (12, 11, 12), (5, 3, 7)])
@pytest.mark.parametrize("nchem", [0, 2, 10])
def test_fp64_small_grids_match_oracle(cuda, shape, nchem):
    torch = cuda
    import gbmv
    bc = (3, 2, 1, 3, 0, 0)
    wl = W.rayleigh_taylor(shape=shape, nchem=nchem, seed=W.SEED_BASE + 704)
    st, ref = O.feuler(wl["fields"], nchem, bc, wl["gamma"], None)
    assert st == 0
    w = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in wl["fields"]]
    out = [torch.full_like(f, np.nan) for f in w]
    assert gbmv.Hydro(shape, nchem, bc, wl["gamma"], None).fEuler(0.0, w, out) == 0
    for a, r in zip(out, ref):
        assert maxnorm_err(a.cpu().numpy(), r) <= 1e-12
