"""The synchronous calls' status and result words: an illegal state or a singular block is reported
by the call that met it and not by the next one, nor by another handle; results are those of the
asynchronous forms (equal bits: the same kernels)."""
import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_illegal_state_is_reported_once(cuda, precision):
    torch = cuda
    import gbmv
    wl = W.rayleigh_taylor(shape=(9, 8, 7), nchem=2, seed=W.SEED_BASE + 730)
    good = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in wl["fields"]]
    bad = [f.clone() for f in good]
    bad[4].view(-1)[5] = -1.0
    out = [torch.empty_like(f) for f in good]
    a, b = (gbmv.Hydro((9, 8, 7), 2, wl["bc"], wl["gamma"], None) for _ in range(2))
    for _ in range(2):
        assert a.fEuler(0.0, bad, out, precision) == -1
        assert b.fEuler(0.0, good, out, precision) == 0
        assert a.fEuler(0.0, good, out, precision) == 0


def test_singular_block_is_reported_once(cuda):
    torch = cuda
    import gbmv
    n = 33
    eye = torch.eye(10, device="cuda", dtype=torch.float64).repeat(n, 1, 1)
    bad = eye.clone()
    bad[17, 3, 3] = 0.0
    ls = gbmv.BlockLinearSolver(n)
    for _ in range(2):
        assert ls.setup(bad.clone().view(-1)) == 1
        assert ls.setup(eye.clone().view(-1)) == 0


def test_norm_forms_agree(cuda):
    torch = cuda
    import gbmv
    wl = W.rayleigh_taylor(shape=(9, 8, 7), nchem=4, seed=W.SEED_BASE + 731)
    y = [torch.from_numpy(np.ascontiguousarray(f)).cuda() for f in wl["fields"]]
    h = gbmv.Hydro((9, 8, 7), 4, wl["bc"], wl["gamma"], None)
    for s in (1e-6, 1e-3):
        v = [s * f for f in y]
        out = torch.zeros(1, device="cuda", dtype=torch.float64)
        norm = h.wrms_norm(v, y, 1e-5, 1e-9)
        h.wrms_norm_async(v, y, 1e-5, 1e-9, out)
        assert norm == out.item()
        mass, energy = h.check_conservation(y)
        assert abs(mass / y[0].sum().item() - 1) < 1e-14
        assert abs(energy / y[4].sum().item() - 1) < 1e-14


def test_more_handles_than_shared_slots(cuda):
    """Handles beyond the shared page's 64 slots, and slots used again after their handle is gone."""
    torch = cuda
    import gbmv
    n = 5
    eye = torch.eye(10, device="cuda", dtype=torch.float64).repeat(n, 1, 1)
    bad = eye.clone()
    bad[2, 7, 7] = 0.0
    for _ in range(2):
        ls = [gbmv.BlockLinearSolver(n) for _ in range(70)]
        for k in (0, 1, 63, 64, 69):
            assert ls[k].setup(bad.clone().view(-1)) == 1
        assert all(x.setup(eye.clone().view(-1)) == 0 for x in ls)
        del ls
