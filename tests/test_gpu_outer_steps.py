"""The float32 Poisson form's accelerated outer iteration
(gpw_poisson_set_acceleration): fewer iterations than plain steps on cubic
grids, grids whose coarsest level its sweeps do not solve and unequal
spacings, to the same stopping test and the same potential."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(N, h, precision):
    from gpawdft_b200.grid_descriptor import GridDescriptor
    from gpawdft_b200.poisson import PoissonSolver
    gd = GridDescriptor(N, tuple(a * b for a, b in zip(N, h)), 0)
    ps = PoissonSolver(nn=3, precision=precision, batch=2)
    ps.set_grid_descriptor(gd)
    ps.initialize()
    return gd, ps


@pytest.mark.parametrize('N,h', [((32, 32, 32), (.38, .38, .38)),
                                 ((48, 40, 56), (.38, .38, .38)),
                                 ((44, 44, 44), (.38, .38, .38)),
                                 ((32, 32, 48), (.38, .43, .35))])
def test_fewer_steps_same_potential(cuda, N, h):
    import torch
    from gpawdft_b200 import _lib
    gd, ps = _solver(N, h, 'fp32')
    rng = np.random.default_rng(1)
    x = [(np.arange(n) + 1.0) / N[c] for c, n in enumerate(gd.n_c)]
    rho = np.zeros((2,) + tuple(gd.n_c))
    for b in range(2):
        for q in (1.0, -1.0, 0.5, -0.5):
            g = [np.exp(-(x[c] - rng.uniform(.3, .7)) ** 2 / .01)
                 for c in range(3)]
            rho[b] += q * np.einsum('i,j,k->ijk', *g)
        rho[b] -= rho[b].mean()
    eps = 1e-20 * (rho ** 2).sum(axis=(1, 2, 3)) * gd.dv
    r = torch.from_numpy(rho).cuda()

    def solve():
        phi = torch.zeros_like(r)
        n = ps.solve_batch(phi, r, eps=eps)
        assert (ps.last_errors <= eps).all()
        return phi.cpu().numpy(), n
    fast, nfast = solve()
    _lib.check(ps._lib.gpw_poisson_set_acceleration(ps._engine[0], 0.0, 0.0))
    plain, nplain = solve()
    assert (nfast < nplain).all(), (nfast, nplain)
    # both stop at a residual of 1e-10 of rho's norm
    assert np.abs(fast - plain).max() < 1e-8 * np.abs(plain).max()


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
