"""The chemistry source, Jacobian and fused Newton over the temperature range and from far and
near carried temperatures, against the oracle: the early end of the temperature iterations, the
floor taken by rounding at table points, the clamped ends of the table.  Tolerances: the parity
bars of the FP64 forms (1e-12 of the largest entry per species and per Jacobian entry); the
interpolation weight carries ~1e-13 in either code, so differences stay near 1e-13."""
import numpy as np
import pytest

import oracle_py as O
import workloads as W

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def _state(n, seed, t_range):
    y, T = W.primordial(n, seed=seed, t_range=t_range)
    return y, T


# (temperature range, carried temperature over the true one; None: 1000 K everywhere); the first
# and last leave the tables' range [1, 1e5] K, where the result is clamped
@pytest.mark.parametrize("t_range,carry", [((0.2, 3.0), 1.0), ((10.0, 1e4), None),
                                           ((10.0, 1e4), 1.0), ((10.0, 1e4), 1.02),
                                           ((3e4, 2e5), 0.9)])
@pytest.mark.parametrize("n", [1, 97, 1500])
def test_source_and_jacobian(cuda, tables, t_range, carry, n):
    torch = cuda
    import gbmv
    y, T = _state(n, 900 + n, t_range)
    oc = O.Chem(tables, y.reshape(-1))
    c = gbmv.Chem(n, tables)
    c.set_scale(_dev(torch, y.reshape(-1)))
    start = np.full(n, 1000.0) if carry is None else T * carry
    oc.Ts[:] = start
    c.state("Ts").copy_(_dev(torch, start))
    z = np.random.default_rng(n).uniform(0.999, 1.001, 10 * n)
    zd = _dev(torch, z)
    f, J = torch.empty_like(zd), torch.empty(100 * n, dtype=torch.float64, device="cuda")
    for _ in range(2):  # the second call from the carried temperature
        fo = oc.rhs(z).reshape(n, 10)
        c.calculate_rhs_cvklu(0.0, zd, f)
        fg = f.cpu().numpy().reshape(n, 10)
        assert np.max(np.abs(c.state("Ts").cpu().numpy() - oc.Ts) / oc.Ts) <= 4e-15
        for s in range(10):
            assert np.max(np.abs(fg[:, s] - fo[:, s])) <= 1e-12 * np.max(np.abs(fo[:, s]))
        Jo = oc.jac(z).reshape(n, 100)
        c.calculate_jacobian_cvklu(0.0, zd, J)
        Jg = J.cpu().numpy().reshape(n, 100)
        for e in range(100):
            assert np.max(np.abs(Jg[:, e] - Jo[:, e])) <= 1e-12 * np.max(np.abs(Jo[:, e])), e


def test_temperature_at_table_points(cuda, tables):
    """Temperatures within an ulp or two of the table points: either neighbouring bin gives the
    same interpolated rates."""
    torch = cuda
    import gbmv
    n = 1024
    y, _ = _state(n, 950, (10.0, 1e4))
    oc = O.Chem(tables, y.reshape(-1))
    c = gbmv.Chem(n, tables)
    c.set_scale(_dev(torch, y.reshape(-1)))
    knots = np.exp(np.arange(n) * (np.log(1e5) / 1023))
    # the Jacobian reads the carried temperature: no solve in between
    for shift in (1.0, 1.0 - 2e-16, 1.0 + 3e-16):
        T = knots * shift
        oc.Ts[:] = T
        oc.dTs_ge[:] = 1e-9
        c.state("Ts").copy_(_dev(torch, T))
        c.state("dTs_ge").copy_(_dev(torch, np.full(n, 1e-9)))
        z = np.ones(10 * n)
        J = torch.empty(100 * n, dtype=torch.float64, device="cuda")
        c.calculate_jacobian_cvklu(0.0, _dev(torch, z), J)
        Jg = J.cpu().numpy().reshape(n, 10, 10)
        Jo = oc.jac(z).reshape(n, 10, 10)
        # the ge column holds slopes, which step from bin to bin: compare the others
        a, b = Jg[:, :9], Jo[:, :9]
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


@pytest.mark.parametrize("precision", [0, 1])
def test_dirk_residency_leaves_results_alone(cuda, tables, precision):
    """The integrator's resident warps follow from the number of cells (lines at 20 and 28 warps of
    cells per SM): the same cells end bit for bit alike in runs of every size."""
    torch = cuda
    import gbmv
    sizes = (1500, 152 * 32 * 20 - 1, 152 * 32 * 20 + 40, 152 * 32 * 28 + 40)
    y, _ = _state(1500, 960, (10.0, 1e4))
    ref = None
    for n in sizes:
        reps = -(-n // 1500)
        scale = np.tile(y, (reps, 1))[:n]
        c = gbmv.Chem(n, tables)
        c.set_scale(_dev(torch, scale.reshape(-1)))
        z = torch.ones(10 * n, dtype=torch.float64, device="cuda")
        assert c.dirk_evolve(0.0, 2e-9, z, 1e11, precision=precision, block=32, rtol=1e-6,
                             atol=1e-10, maxcor=10, nlscoef=0.01) == 0
        z = z.view(n, 10)
        if ref is None:
            ref = z
        for k in range(0, n, 1500):
            m = min(1500, n - k)
            assert torch.equal(z[k:k + m], ref[:m])
