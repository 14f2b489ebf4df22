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


def test_interval():
    def ops(N, h=(1, 1, 1)):
        gd = GridDescriptor((N,) * 3, tuple(N * a for a in h), 0)
        out = [laplace(gd, NN3)]
        while True:
            try:
                gd = gd.coarsen()
            except ValueError:
                return out
            out.append(laplace(gd, [-2.0, 1.0]))
    lo, hi = inner_spectrum(ops(64))
    assert 0.77 < lo < 0.79 and hi == 1.045      # Arnoldi: 0.794 .. 1.042
    # unequal spacings (Arnoldi: 0.679 .. 1.056), and a 25-point coarsest level
    assert inner_spectrum(ops(32, (1, 1.15, .9)))[0] < 0.68
    lo, hi = inner_spectrum(ops(100))
    assert lo < 0.4 and hi > 1.6
