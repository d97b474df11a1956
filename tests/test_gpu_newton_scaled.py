"""The fused Newton's two ways to its matrix: with every column scaled by its own variable, and plain
where a variable is zero or far from 1.  Against the separate Jacobian's system solved in extended
precision, the error of a cell measured over its variables.  Partial pivoting on rows whose scales
differ by many decades has no useful bound for the worst cell, so the bars are on the median and the
90th percentile: ~eps times conditions up to 1e3 and 1e5 for the FP64 factor and the refined FP32
one, and 2^-24 in eps' place without refinement."""
import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu

TU, GAMMA, N = 1.0e11, 1e-4, 1500


def _solve(A, b):
    """Extended-precision elimination of a batch of equilibrated systems."""
    A, b = A.astype(np.longdouble), b.astype(np.longdouble)
    s = 1 / np.abs(A).max(2)
    A, b = A * s[:, :, None], b * s
    cells, m = np.arange(len(b)), b.shape[1]
    for k in range(m):
        p = k + np.abs(A[:, k:, k]).argmax(1)
        A[cells, p], A[:, k] = A[:, k].copy(), A[cells, p].copy()
        b[cells, p], b[:, k] = b[:, k].copy(), b[cells, p].copy()
        for r in range(k + 1, m):
            f = A[:, r, k] / A[:, k, k]
            A[:, r] -= f[:, None] * A[:, k]
            b[:, r] -= f * b[:, k]
    for k in range(m - 1, -1, -1):
        b[:, k] = (b[:, k] - (A[:, k, k + 1:] * b[:, k + 1:]).sum(1)) / A[:, k, k]
    return b


def _errors(torch, tables, decades, zeros, lu, refine):
    import gbmv
    y, T = W.primordial(N, seed=W.SEED_BASE + 740)
    rng = np.random.default_rng(5)
    z = 10.0 ** rng.uniform(-decades, decades, (N, 10))
    scale = y / z
    for _ in range(zeros):
        z[np.arange(N), rng.integers(0, 8, N)] = 0.0

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()

    c = gbmv.Chem(N, tables)
    c.set_scale(dev(scale))
    c.state("Ts").copy_(dev(T))
    zd = dev(z)
    f, x = torch.full_like(zd, np.nan), torch.full_like(zd, np.nan)
    assert c.newton_iteration(0.0, zd, f, x, GAMMA, TU, lu_precision=lu, refine=refine) == 0
    J = torch.empty(100 * N, dtype=torch.float64, device="cuda")
    c.calculate_jacobian_cvklu(0.0, zd, J, TU)
    J = J.cpu().numpy().reshape(N, 10, 10).transpose(0, 2, 1).astype(np.longdouble)
    ref = _solve(np.eye(10) - np.longdouble(GAMMA) * J, f.cpu().numpy().reshape(N, 10))
    x = x.cpu().numpy().reshape(N, 10)
    assert np.isfinite(x).all()
    unit = np.where(z == 0.0, np.abs(ref) + np.longdouble(1e-300), np.abs(z))
    err = (np.abs(x - ref) / unit).max(1) / (np.abs(ref) / unit).max(1)
    return np.quantile(err.astype(np.float64), [0.5, 0.9])


@pytest.mark.parametrize("decades,zeros", [(0, 0), (3, 0), (6, 0), (0, 1), (0, 2), (3, 1)])
@pytest.mark.parametrize("lu,refine", [(0, 0), (1, 2), (1, 4)])
def test_newton_with_variables_away_from_one(cuda, tables, decades, zeros, lu, refine):
    median, most = _errors(cuda, tables, decades, zeros, lu, refine)
    assert median <= 2.2e-13 and most <= 2.2e-11


@pytest.mark.parametrize("decades", [0, 3, 6, 10])
def test_newton_without_refinement(cuda, tables, decades):
    """The FP32 factor alone."""
    median, most = _errors(cuda, tables, decades, 0, 1, 0)
    assert median <= 6e-5 and most <= 6e-3


def test_newton_without_refinement_far_from_one(cuda, tables):
    """Variables over 56 decades: scaled columns of the FP32 factor would leave the float range (all
    digits of the median cell lost), the plain ones keep some of them."""
    assert _errors(cuda, tables, 28, 0, 1, 0)[0] <= 1e-2
