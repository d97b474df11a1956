"""Block LU tiles: block counts around the 32-block tile and the persistent grid (1216 factor, 1064
solve CTAs), arrays that are only 8-byte aligned, pivoting.  Against LAPACK (numpy); well-
conditioned random blocks, so a solution's relative error is bounded by ~10 n eps cond ~ 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 1217, 34049, 38913])
@pytest.mark.parametrize("offset", [0, 1])
def test_block_lu_tiles(cuda, n, offset):
    torch = cuda
    import gbmv
    rng = np.random.default_rng(n)
    J = rng.uniform(-1.0, 1.0, size=(n, 10, 10))  # [block][col][row]
    J[:, np.arange(10), np.arange(10)] *= 0.1      # weak diagonals: rows are interchanged
    gamma = 0.7
    M = np.eye(10) - gamma * J.transpose(0, 2, 1)
    b = rng.standard_normal((n, 10))

    def dev(a):  # at an address 8 bytes past a 16-byte boundary when offset is 1
        buf = torch.empty(a.size + 2, dtype=torch.float64, device="cuda")
        v = buf[offset:offset + a.size]
        v.copy_(torch.from_numpy(a.reshape(-1)))
        return v

    A, B, X = dev(J), dev(b), dev(np.zeros_like(b))
    gbmv.form_newton_matrix(A, gamma)
    assert np.allclose(A.cpu().numpy().reshape(n, 10, 10), M.transpose(0, 2, 1), rtol=4e-16,
                       atol=4e-16)
    ls = gbmv.BlockLinearSolver(n)
    assert ls.setup(A) == 0
    ls.solve(A, X, B)
    ref = np.linalg.solve(M, b[:, :, None])[:, :, 0]
    cond = np.linalg.cond(M)
    err = np.abs(X.cpu().numpy().reshape(n, 10) - ref).max(1) / np.abs(ref).max(1)
    assert np.all(err <= 1e-14 * cond + 1e-14)


def test_block_lu_nan_and_zero_blocks(cuda):
    """A NaN entry stays in its block; a zero pivot is reported."""
    torch = cuda
    import gbmv
    M = np.tile(np.eye(10) * 2.0, (40, 1, 1))
    M[7, 3, 5] = np.nan
    A = torch.from_numpy(M.reshape(-1)).cuda()
    ls = gbmv.BlockLinearSolver(40)
    assert ls.setup(A) == 0
    x = torch.empty(400, dtype=torch.float64, device="cuda")
    ls.solve(A, x, torch.ones(400, dtype=torch.float64, device="cuda"))
    good = np.delete(x.cpu().numpy().reshape(40, 10), 7, axis=0)
    assert np.array_equal(good, np.full((39, 10), 0.5))
