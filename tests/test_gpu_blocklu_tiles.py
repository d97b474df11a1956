"""The block solve at the ends of its persistent grid (608 CTAs, tiles of 32 blocks, the next tile in
flight while one is solved): a CTA's second and third tile, of one block and whole, and the solution
written over the right-hand side.  Against LAPACK (numpy): ~10 n eps times the block's condition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = 608 * 32


@pytest.mark.parametrize("n", [31, 33, GRID - 1, GRID, GRID + 1, GRID + 32, 2 * GRID, 2 * GRID + 1])
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
def test_solve_at_the_ends_of_the_grid(cuda, n, in_place, offset):
    torch = cuda
    import gbmv
    rng = np.random.default_rng(n)
    M = rng.uniform(-1.0, 1.0, size=(n, 10, 10))
    M[:, np.arange(10), np.arange(10)] *= 0.1  # weak diagonals: rows are interchanged
    b = rng.standard_normal((n, 10))

    def dev(a):  # at an address 8 bytes past a 16-byte boundary when offset is 1
        buf = torch.empty(a.size + 2, dtype=torch.float64, device="cuda")
        v = buf[offset:offset + a.size]
        v.copy_(torch.from_numpy(np.ascontiguousarray(a).reshape(-1)))
        return v

    A, B = dev(M.transpose(0, 2, 1)), dev(b)
    X = B if in_place else dev(np.full_like(b, np.nan))
    ls = gbmv.BlockLinearSolver(n)
    assert ls.setup(A) == 0
    ls.solve(A, X, B)
    ref = np.linalg.solve(M, b[:, :, None])[:, :, 0]
    err = np.abs(X.cpu().numpy().reshape(n, 10) - ref).max(1) / np.abs(ref).max(1)
    assert np.all(err <= 1e-14 * np.linalg.cond(M) + 1e-14)
    if not in_place:
        assert np.array_equal(B.cpu().numpy().reshape(n, 10), b)
