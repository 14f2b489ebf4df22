"""The float32 Poisson form's accelerated outer iteration
(gpw_poisson_set_acceleration): fewer iterations than plain steps on cubic
grids, grids whose coarsest level its sweeps do not solve and unequal
spacings, to the same stopping test and the same potential; and the return to
plain steps where an interval does not hold the spectrum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(N, h, precision, **kwargs):
    from gpawdft_b200.grid_descriptor import GridDescriptor
    from gpawdft_b200.poisson import PoissonSolver
    gd = GridDescriptor(N, tuple(a * b for a, b in zip(N, h)), 0)
    ps = PoissonSolver(nn=3, precision=precision, batch=2, **kwargs)
    ps.set_grid_descriptor(gd)
    ps.initialize()
    return gd, ps


def _charges(gd, N):
    rng = np.random.default_rng(1)
    x = [(np.arange(n) + 1.0) / N[c] for c, n in enumerate(gd.n_c)]
    rho = np.zeros((2,) + tuple(gd.n_c))
    for b in range(2):
        for q in (1.0, -1.0, 0.5, -0.5):
            g = [np.exp(-(x[c] - rng.uniform(.3, .7)) ** 2 / .01)
                 for c in range(3)]
            rho[b] += q * np.einsum('i,j,k->ijk', *g)
        rho[b] -= rho[b].mean()
    return rho


def _solve(ps, rho, interval=None):
    """Potentials and iterations to a residual of 1e-10 of rho's norm."""
    import torch
    from gpawdft_b200 import _lib
    if interval is not None:
        _lib.check(ps._lib.gpw_poisson_set_acceleration(ps._engine[0],
                                                        *interval))
    eps = 1e-20 * (rho ** 2).sum(axis=(1, 2, 3)) * ps.gd.dv
    r = torch.from_numpy(rho).cuda()
    phi = torch.zeros_like(r)
    n = ps.solve_batch(phi, r, eps=eps)
    assert (ps.last_errors <= eps).all()
    return phi.cpu().numpy(), n


def _same(a, b):
    # both stop at a residual of 1e-10 of rho's norm
    return np.abs(a - b).max() < 1e-8 * np.abs(b).max()


@pytest.mark.parametrize('N,h,levels', [
    ((32, 32, 32), (.38, .38, .38), None),
    ((48, 40, 56), (.38, .38, .38), None),
    ((44, 44, 44), (.38, .38, .38), None),
    ((32, 32, 48), (.38, .43, .35), None),
    # a coarsest level of 47^3 points: an interval clamped at hi / 16
    ((96, 96, 96), (.38, .38, .38), 2)])
@pytest.mark.filterwarnings('ignore')
def test_fewer_steps_same_potential(cuda, N, h, levels):
    gd, ps = _solver(N, h, 'fp32', max_levels=levels)
    rho = _charges(gd, N)
    fast, nfast = _solve(ps, rho)
    plain, nplain = _solve(ps, rho, (0.0, 0.0))
    assert (nfast < nplain).all(), (nfast, nplain)
    assert _same(fast, plain)


def test_interval_around_one(cuda):
    """Equally far to both sides of 1: the first length of its cycle is 1."""
    N = (32, 32, 32)
    gd, ps = _solver(N, (.38,) * 3, 'fp32')
    rho = _charges(gd, N)
    fast, nfast = _solve(ps, rho, (0.8, 1.2))
    plain, nplain = _solve(ps, rho, (0.0, 0.0))
    assert (nfast < nplain).all(), (nfast, nplain)
    assert _same(fast, plain)


def test_back_to_plain_steps(cuda):
    """The V-cycle's spectrum (0.79 .. 1.04) lies far above the interval: the
    first two steps amplify every mode 5 and 2.4 times, the second growth is
    seen, and plain steps (0.21 a step) go on from there.  The next solve
    starts with accelerated steps again."""
    N = (32, 32, 32)
    gd, ps = _solver(N, (.38,) * 3, 'fp32')
    rho = _charges(gd, N)
    plain, nplain = _solve(ps, rho, (0.0, 0.0))
    for _ in range(2):
        phi, n = _solve(ps, rho, (0.02, 0.3))
        assert (n > nplain).all() and (n <= nplain + 6).all(), (n, nplain)
        assert _same(phi, plain)
    phi, n = _solve(ps, rho, (0.78, 1.045))
    assert (n < nplain).all(), (n, nplain)
    assert _same(phi, plain)


def test_solve_many_takes_new_settings(cuda):
    """Several engines in one graph: a changed interval reaches the next
    solve, and engines made after others of the same sizes were freed have
    graphs of their own."""
    from gpawdft_b200 import _lib
    from gpawdft_b200.poisson import solve_many
    counts = []
    for _ in range(3):
        pairs = [_solver((N,) * 3, (.38,) * 3, 'fp32') for N in (32, 40)]
        rhos = [_charges(gd, gd.N_c) for gd, ps in pairs]
        eps = [1e-20 * (r ** 2).sum(axis=(1, 2, 3)) * gd.dv
               for r, (gd, ps) in zip(rhos, pairs)]

        def solve():
            phis = [np.zeros_like(r) for r in rhos]
            return phis, solve_many([ps for gd, ps in pairs], phis, rhos, eps)
        fast, nfast = solve()
        for gd, ps in pairs:
            _lib.check(ps._lib.gpw_poisson_set_acceleration(ps._engine[0],
                                                            0.0, 0.0))
        plain, nplain = solve()
        for a, b, n, m in zip(fast, plain, nfast, nplain):
            assert (n < m).all(), (n, m)
            assert _same(a, b)
        counts.append(np.concatenate(nfast + nplain))
        for gd, ps in pairs:
            ps._free_engine()
    assert np.array_equal(counts[0], counts[1])
    assert np.array_equal(counts[0], counts[2])


def test_rejects_bad_intervals(cuda):
    from gpawdft_b200 import _lib
    lib = _lib.load()
    gd, ps = _solver((16, 16, 16), (.38, .38, .38), 'fp32')
    h = ps._engine[0]
    assert lib.gpw_poisson_set_acceleration(None, .5, 1.) == _lib.GPW_EINVAL
    assert lib.gpw_poisson_set_acceleration(h, 0.0, 1.0) == _lib.GPW_EINVAL
    assert lib.gpw_poisson_set_acceleration(h, -1.0, 1.0) == _lib.GPW_EINVAL
    assert lib.gpw_poisson_set_acceleration(h, .5, float('nan')) == \
        _lib.GPW_EINVAL
    assert lib.gpw_poisson_set_acceleration(h, 0.8, 1.05) == _lib.GPW_OK
