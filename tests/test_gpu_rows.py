"""The whole-row star stencil (gpw_rows.cuh), pinned, against the oracle
(c/operators.c apply over the c/bc.c halo, restated).

Shapes sit at its edges: rows of odd length (element-wise staging) and of
whole 16-byte units (one bulk copy), a single tile, a tile longer than the
grid, a last tile with part of its rows, fewer rows than the stencil reaches,
one-point axes, more planes per CTA than the grid has (several segments) and
fewer.  Every mix of periodic and zero axes, Bloch phases, gradients (which
stage no halo planes or rows), the potential term, and the small-grid kernel
(gpw_direct.cuh) on the same inputs.  Tolerances as for the other stencils."""
import numpy as np
import pytest

from helpers import TOL, oracle_dtype, rand, relerr
from oracle import layer as ol
from oracle.geometry import GridDescriptor as OGD, phase_cd_for_k

pytestmark = pytest.mark.gpu

DTYPES = [np.complex128, np.complex64, np.float64, np.float32]
PBCS = [(1, 1, 1), (0, 0, 0), (1, 0, 1), (0, 1, 0), (0, 0, 1)]
SHAPES = [(7, 9, 11), (16, 8, 20), (5, 33, 95), (40, 3, 96), (6, 50, 17),
          (9, 4, 128), (3, 3, 3), (4, 11, 200)]


@pytest.fixture
def pin():
    from gpawdft_b200 import _lib
    lib = _lib.load()
    yield lambda k: _lib.check(lib.gpw_set_bloch_layout(k))
    _lib.check(lib.gpw_set_bloch_layout(0))


def _setup(n, pbc):
    from gpawdft_b200.grid_descriptor import GridDescriptor
    N = tuple(m if p else m + 1 for m, p in zip(n, pbc))
    cell = tuple(0.2 * m for m in N)
    return GridDescriptor(N, cell, pbc), OGD(N, cell, pbc)


def _phases(ogd, dtype, seed):
    if np.dtype(dtype).kind != 'c':
        return None
    return phase_cd_for_k(ogd, np.random.default_rng(seed).uniform(-.5, .5, 3))


@pytest.mark.parametrize('layout', [15, 16, 0])
@pytest.mark.parametrize('dtype', DTYPES)
@pytest.mark.parametrize('pbc', PBCS)
@pytest.mark.parametrize('n', SHAPES)
def test_apply(cuda, pin, n, pbc, dtype, layout):
    import gpawdft_b200.fd_operators as fd
    gd, ogd = _setup(n, pbc)
    a = rand((3,) + tuple(gd.n_c), dtype, 1)
    ph = _phases(ogd, dtype, 2)
    pin(layout)
    ops = [(lambda m, g, d: m.Laplace(g, -0.5, 3, d)),
           (lambda m, g, d: m.Laplace(g, -0.5, 1, d)),
           (lambda m, g, d: m.Gradient(g, 0, 1.0, 2, d)),
           (lambda m, g, d: m.Gradient(g, 1, 1.0, 3, d)),
           (lambda m, g, d: m.Gradient(g, 2, 1.0, 3, d))]
    for make in ops:
        out = np.zeros_like(a)
        make(fd, gd, dtype).apply(a, out, ph)
        ref = np.zeros(a.shape, oracle_dtype(dtype))
        make(ol, ogd, oracle_dtype(dtype)).apply(
            a.astype(oracle_dtype(dtype)), ref, ph)
        assert relerr(out, ref) < TOL[np.dtype(dtype)]


@pytest.mark.parametrize('layout', [15, 16, 0])
@pytest.mark.parametrize('dtype', DTYPES)
@pytest.mark.parametrize('n,pbc', [((9, 21, 31), (0, 0, 0)),
                                   ((12, 10, 16), (1, 1, 1))])
def test_potential(cuda, pin, n, pbc, dtype, layout):
    from gpawdft_b200.fd_operators import Laplace
    gd, ogd = _setup(n, pbc)
    a = rand((5,) + tuple(gd.n_c), dtype, 3)
    real = np.float64 if np.dtype(dtype) in (np.dtype(np.float64),
                                             np.dtype(complex)) \
        else np.float32
    v = rand(tuple(gd.n_c), real, 4)
    ph = _phases(ogd, dtype, 5)
    pin(layout)
    out = np.zeros_like(a)
    Laplace(gd, -0.5, 3, dtype).apply_potential(a, out, v, ph)
    wide = a.astype(oracle_dtype(dtype))
    ref = np.zeros_like(wide)
    ol.Laplace(ogd, -0.5, 3, oracle_dtype(dtype)).apply(wide, ref, ph)
    ref += wide * v
    assert relerr(out, ref) < TOL[np.dtype(dtype)]


@pytest.mark.parametrize('pbc', [(0, 0, 0), (1, 1, 1)])
@pytest.mark.parametrize('dtype', [np.float64, np.complex128, np.float32])
def test_many_bands_past_l2(cuda, pin, pbc, dtype):
    """More units than CTAs and several segments each: equal to the pinned
    kernel run band by band (every output sums its terms in one order)."""
    import torch
    from gpawdft_b200.fd_operators import Laplace
    gd, ogd = _setup((20, 30, 47), pbc)
    a = torch.from_numpy(rand((200,) + tuple(gd.n_c), dtype, 6)).cuda()
    ph = _phases(ogd, dtype, 7)
    op = Laplace(gd, -0.5, 3, dtype)
    pin(15)
    out = torch.empty_like(a)
    op.apply(a, out, ph)
    for b in (0, 1, 99, 199):
        one = torch.empty_like(a[b])
        op.apply(a[b], one, ph)
        assert torch.equal(out[b], one)


@pytest.mark.parametrize('dtype', DTYPES)
@pytest.mark.parametrize('n,pbc', [((9, 10, 31), (1, 1, 1)),
                                   ((18, 33, 65), (1, 1, 1)),
                                   ((9, 50, 180), (0, 1, 1)),
                                   ((21, 6, 32), (1, 0, 0)),
                                   ((5, 7, 250), (1, 1, 1))])
@pytest.mark.parametrize('skew,mb', [(0, 9), (1, 9), (0, 4.5), (0, 2.5)])
@pytest.mark.parametrize('nn', [1, 3])
def test_gradients_by_rule(cuda, n, pbc, dtype, skew, mb, nn):
    """Gradients of grids without a tuned layout to both sides of the sizes at
    which the rule sends them to the whole-row kernel, with rows too long for
    it and (but complex128) grids that start off a 16-byte boundary."""
    import torch
    from gpawdft_b200.fd_operators import Gradient
    gd, ogd = _setup(n, pbc)
    if np.dtype(dtype) == np.dtype(complex):
        skew = 0
    nin = int(mb * 2 ** 20 / (int(np.prod(n)) * np.dtype(dtype).itemsize)) + 1
    size = nin * int(np.prod(n))
    flat = torch.from_numpy(rand((size + skew,), dtype, 8)).cuda()
    a = flat[skew:].view((nin,) + tuple(gd.n_c))
    ends = a[[0, -1]].cpu().numpy().astype(oracle_dtype(dtype))
    ph = _phases(ogd, dtype, 9)
    for axis in range(3):
        out = torch.empty_like(a)
        Gradient(gd, axis, 1.0, nn, dtype).apply(a, out, ph)
        ref = np.zeros_like(ends)
        ol.Gradient(ogd, axis, 1.0, nn, oracle_dtype(dtype)).apply(ends, ref,
                                                                   ph)
        assert relerr(out[[0, -1]].cpu().numpy(), ref) < TOL[np.dtype(dtype)]
