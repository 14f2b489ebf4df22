"""Stencil symbols (poisson.jacobi_spectrum): the per-axis sum that star
stencils take against the symbol evaluated point by point, and the interval
of the accelerated outer iteration."""
import numpy as np
import pytest

from gpawdft_b200.grid_descriptor import GridDescriptor
from gpawdft_b200.poisson import inner_spectrum, jacobi_spectrum


class Stencil:
    def __init__(self, gd, coef, offs):
        self.gd = gd
        self.coef_p = np.asarray(coef, float)
        self.offset_pc = np.asarray(offs, int).reshape(-1, 3)


def laplace(gd, table):
    coef, offs = [0.0], [(0, 0, 0)]
    for c in range(3):
        h = gd.h_cv[c, c]
        coef[0] += table[0] / h ** 2
        for s, w in enumerate(table[1:], 1):
            for t in (s, -s):
                o = [0, 0, 0]
                o[c] = t
                offs.append(o)
                coef.append(w / h ** 2)
    return Stencil(gd, -np.array(coef), offs)


NN3 = [-49 / 18, 3 / 2, -3 / 20, 1 / 90]


@pytest.mark.parametrize('pbc', [0, 1, (1, 0, 1)])
@pytest.mark.parametrize('N', [(4, 4, 4), (12, 10, 14)])
def test_star_symbol(N, pbc):
    gd = GridDescriptor(N, tuple(0.3 * n for n in N), pbc)
    op = laplace(gd, NN3)
    t = [2 * np.pi * np.arange(n) / n if p else
         np.pi * np.arange(1, n + 1) / (n + 1)
         for n, p in zip(gd.n_c, gd.pbc_c)]
    g = np.meshgrid(*t, indexing='ij')
    lam = sum(c * np.cos(sum(a * b for a, b in zip(o, g)))
              for c, o in zip(op.coef_p, op.offset_pc)) / op.coef_p[0]
    # 19 terms of at most 1, summed in another order
    assert abs(jacobi_spectrum(op) - lam.max()) < 19 * 2.0 ** -52 * lam.max()
    low = lam[lam > 1e-12 * lam.max()].min()
    assert abs(jacobi_spectrum(op, lowest=True) - low) < 19 * 2.0 ** -50


def ops(N, h=(1, 1, 1), pbc=0, levels=9):
    N = (N,) * 3 if isinstance(N, int) else N
    gd = GridDescriptor(N, tuple(n * a for n, a in zip(N, h)), pbc)
    out = [laplace(gd, NN3)]
    while len(out) < levels:
        try:
            gd = gd.coarsen()
        except ValueError:
            break
        out.append(laplace(gd, [-2.0, 1.0]))
    return out


def test_interval():
    lo, hi = inner_spectrum(ops(64))
    assert 0.77 < lo < 0.79 and hi == 1.045      # Arnoldi: 0.794 .. 1.042
    # unequal spacings (Arnoldi: 0.679 .. 1.056), and a 25-point coarsest level
    assert inner_spectrum(ops(32, (1, 1.15, .9)))[0] < 0.68
    lo, hi = inner_spectrum(ops(100))
    assert lo < 0.4 and hi > 1.6


@pytest.mark.parametrize('case', [
    dict(N=202), dict(N=354), dict(N=362), dict(N=400, levels=2),
    dict(N=(16, 16, 1202), pbc=1)])
def test_interval_of_hard_grids(case):
    """Coarsest levels that their sweeps hardly solve: the engine takes the
    interval (0 < lo < hi), and no cycle of the five step lengths amplifies a
    mode up to 1.06 hi on its way, in the order that the engine takes them."""
    lo, hi = inner_spectrum(ops(**case))
    assert 0.0 < lo < hi <= 2.0
    lam = np.linspace(0.0, 1.06 * hi, 20001)[1:]
    p = np.ones_like(lam)
    for j in (2, 0, 4, 1, 3):
        node = 0.5 * (hi + lo) + 0.5 * (hi - lo) * np.cos((2 * j + 1) *
                                                          np.pi / 10)
        p = p * (1.0 - lam / node)
        assert np.abs(p).max() <= 1.0
