"""The cell-staged star stencil (gpw_star_cells.cuh) against the oracle
(c/operators.c apply, c/bmgs/relax.c, c/bmgs/fd.c restated): batches just past
the size up to which the small-grid kernel serves (8 MB of input), with rows
of odd length (one element a cell) and of whole 16-byte units, partial tiles
in both axes and every tile, every radius, every mix of periodic and
zero axes, Bloch phases, and the potential, aux, residual and Jacobi
epilogues.  The first and last members are compared; tolerances as for the
other stencils (float32 sums of squares: 1e-6)."""
import numpy as np
import pytest

from helpers import TOL, oracle_dtype, rand, relerr
from oracle import layer as ol
from oracle.geometry import GridDescriptor as OGD, phase_cd_for_k

pytestmark = pytest.mark.gpu

DTYPES = [np.complex128, np.complex64, np.float64, np.float32]
CASES = [((23, 49, 51), (0, 0, 0)), ((23, 49, 51), (1, 1, 1)),
         ((9, 45, 64), (1, 1, 1)), ((21, 35, 96), (0, 1, 1)),
         ((12, 130, 33), (1, 0, 1)), ((11, 19, 22), (1, 1, 0)),
         ((9, 47, 67), (0, 1, 1))]


def _setup(n, pbc, dtype, seed):
    from gpawdft_b200.grid_descriptor import GridDescriptor
    import torch
    N = tuple(m if p else m + 1 for m, p in zip(n, pbc))
    cell = tuple(0.2 * m for m in N)
    gd, ogd = GridDescriptor(N, cell, pbc), OGD(N, cell, pbc)
    nin = 9 * 2 ** 20 // (int(np.prod(n)) * np.dtype(dtype).itemsize) + 1
    ends = rand((2,) + n, dtype, seed)
    a = torch.from_numpy(rand((nin,) + n, np.dtype(dtype), seed + 1)).cuda()
    a[0] = torch.from_numpy(ends[0]).cuda()
    a[-1] = torch.from_numpy(ends[1]).cuda()
    ph = None
    if np.dtype(dtype).kind == 'c':
        ph = phase_cd_for_k(ogd, np.random.default_rng(seed).uniform(-.5, .5,
                                                                     3))
    return gd, ogd, a, ends, ph


def _ends(t):
    return np.stack([t[0].cpu().numpy(), t[-1].cpu().numpy()])


def _apply(op, ends, dtype, ph):
    wide = ends.astype(oracle_dtype(dtype))
    ref = np.zeros_like(wide)
    op.apply(wide, ref, ph)
    return ref


@pytest.mark.parametrize('nn', [1, 2, 3, 4])
@pytest.mark.parametrize('dtype', DTYPES)
@pytest.mark.parametrize('n,pbc', CASES)
def test_apply_with_terms(cuda, n, pbc, dtype, nn):
    import torch
    from gpawdft_b200.fd_operators import Laplace
    gd, ogd, a, ends, ph = _setup(n, pbc, dtype, 10 * nn)
    op = Laplace(gd, -0.5, nn, dtype)
    ref = _apply(ol.Laplace(ogd, -0.5, nn, oracle_dtype(dtype)), ends, dtype,
                 ph)
    tol = TOL[np.dtype(dtype)]
    out = torch.empty_like(a)
    op.apply(a, out, ph)
    assert relerr(_ends(out), ref) < tol
    real = np.float64 if np.dtype(dtype).itemsize == 8 * (1 + (
        np.dtype(dtype).kind == 'c')) else np.float32
    v = rand(n, real, 5)
    op.apply_potential(a, out, torch.from_numpy(v).cuda(), ph)
    assert relerr(_ends(out), ref + ends * v) < tol
    op.apply_fused(a, out, ph, vt_g=torch.from_numpy(v).cuda(), aux=a,
                   aux_scale=0.75)
    assert relerr(_ends(out), ref + ends * v + 0.75 * ends) < tol


@pytest.mark.parametrize('nn', [1, 2, 3, 4])
@pytest.mark.parametrize('dtype', [np.float64, np.float32])
@pytest.mark.parametrize('n,pbc', CASES)
def test_residual_and_jacobi(cuda, n, pbc, dtype, nn):
    import torch
    from gpawdft_b200.fd_operators import Laplace
    gd, ogd, f, ends, _ = _setup(n, pbc, dtype, 20 * nn)
    s = torch.from_numpy(rand(tuple(f.shape), dtype, 6)).cuda()
    op = Laplace(gd, -0.25 / np.pi, nn, dtype)
    oop = ol.Laplace(ogd, -0.25 / np.pi, nn)
    src = _ends(s).astype(float)
    want = _apply(oop, ends, dtype, None) - src
    r = torch.empty_like(f)
    norm = op.residual(f, s, r)
    assert relerr(_ends(r), want) < TOL[np.dtype(dtype)]
    got = norm.cpu().numpy()[[0, -1]]
    sq = (want ** 2).sum(axis=(1, 2, 3))
    assert np.abs(got - sq).max() < \
        (1e-12 if np.dtype(dtype) == np.float64 else 1e-6) * sq.max()
    g = f.clone()
    op.relax(2, g, s, 3, 0.7)
    for k in range(2):
        x = ends[k].astype(float)
        oop.relax(2, x, src[k], 3, 0.7)
        assert relerr(_ends(g)[k], x) < 4 * TOL[np.dtype(dtype)]


@pytest.mark.parametrize('nn', [1, 2, 3])
@pytest.mark.parametrize('dtype', [np.complex128, np.complex64])
@pytest.mark.parametrize('slope', [-1, 1])
@pytest.mark.parametrize('n,pbc', [((20, 20, 33), (1, 1, 1)),
                                   ((9, 9, 64), (1, 1, 0)),
                                   ((37, 37, 12), (0, 0, 1)),
                                   ((6, 6, 6), (1, 1, 1))])
def test_star_and_one_diagonal(cuda, n, pbc, slope, dtype, nn):
    """Hexagonal cells (both angles) of complex grids: the diagonal of axes 0
    and 1 with the star, corners past one and two boundaries."""
    import torch
    from gpawdft_b200.fd_operators import Laplace
    from gpawdft_b200.grid_descriptor import GridDescriptor
    N = tuple(m if p else m + 1 for m, p in zip(n, pbc))
    a = 0.2 * N[0]
    cell = [(a, 0, 0), (slope * -0.5 * a, 0.75 ** 0.5 * a, 0),
            (0, 0, 0.2 * N[2])]
    gd, ogd = GridDescriptor(N, cell, pbc), OGD(N, cell, pbc)
    x = rand((3,) + n, dtype, 31 * nn)
    v = rand(n, np.float64 if dtype == np.complex128 else np.float32, 5)
    ph = phase_cd_for_k(ogd, np.array([0.13, -0.31, 0.22]))
    tol = TOL[np.dtype(dtype)]
    dev, vt = torch.from_numpy(x).cuda(), torch.from_numpy(v).cuda()
    out = torch.empty_like(dev)
    op = Laplace(gd, -0.5, nn, dtype)
    ref = _apply(ol.Laplace(ogd, -0.5, nn, oracle_dtype(dtype)), x, dtype, ph)
    op.apply(dev, out, ph)
    assert relerr(out.cpu().numpy(), ref) < tol
    op.apply_fused(dev, out, ph, vt_g=vt, aux=dev, aux_scale=0.75)
    assert relerr(out.cpu().numpy(), ref + x * v + 0.75 * x) < tol
    op.apply_potential(dev, out, vt, ph)
    assert relerr(out.cpu().numpy(), ref + x * v) < tol


def _rows_of_five_points(op, a, n):
    """(row, the sum of the five points in the plane) at rows of a."""
    import torch
    c = {tuple(o): w for o, w in zip(op.offset_pc, op.coef_p)}
    for y in (0, 1, n // 2, n - 40, n - 1):
        rows = torch.nn.functional.pad(a[0, max(0, y - 1):y + 2],
                                       (1, 1, int(y == 0), int(y == n - 1)))
        yield y, c[0, 0, 0] * rows[1, 1:-1] + \
            c[0, 0, 1] * (rows[1, 2:] + rows[1, :-2]) + \
            c[0, 1, 0] * (rows[0, 1:-1] + rows[2, 1:-1])


@pytest.mark.parametrize('dtype,N', [(complex, 16500), (float, 23300)])
def test_planes_past_32_bits(cuda, dtype, N):
    """Planes of more than 4 GiB with rows off the 16-byte boundaries of the
    TMA kernel: applies, and the residual with its norm."""
    import torch
    from gpawdft_b200.fd_operators import Laplace
    from gpawdft_b200.grid_descriptor import GridDescriptor
    gd = GridDescriptor((2, N, N), (0.4, 0.2 * N, 0.2 * N), 0)
    n = N - 1
    assert n * n * np.dtype(dtype).itemsize > 2 ** 32
    torch.manual_seed(1)
    a = torch.randn((1, n, n), device='cuda', dtype=torch.complex128
                    if dtype is complex else torch.float64)
    op = Laplace(gd, -0.5, 1, dtype)
    out = torch.empty_like(a)
    op.apply(a, out, None if dtype is float else np.ones((3, 2), complex))
    for y, ref in _rows_of_five_points(op, a, n):
        err = (out[0, y] - ref).abs().max() / ref.abs().max()
        assert err < TOL[np.dtype(dtype)], (y, err)
    if dtype is float:
        norm = op.residual(a[None], a[None], out[None])
        for y, ref in _rows_of_five_points(op, a, n):
            ref = ref - a[0, y]
            err = (out[0, y] - ref).abs().max() / ref.abs().max()
            assert err < TOL[np.dtype(dtype)], (y, err)
        want = (out * out).sum()
        assert (norm[0] - want).abs() < 1e-12 * want
