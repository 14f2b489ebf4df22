"""The matrix of pair integrals on the tensor-core kernel (gpw_pairs.cu)
against NumPy in 64 bits, at the edges of its 8 x 8 blocks, warp tiles and
point ranges, for every element type; and few pairs of long vectors, which
take a reduction each.

Bound: a sum of n products in float64, in any order, is off by at most
n 2^-53 sum |a| |b| (complex: four real products per term)."""
import numpy as np
import pytest

from helpers import rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [np.float64, np.complex128, np.float32,
                                   np.complex64])
@pytest.mark.parametrize('nx,ny,N', [(1, 2, (1, 1, 1)), (2, 1, (3, 1, 1)),
                                     (7, 9, (4, 4, 4)), (8, 8, (5, 7, 9)),
                                     (24, 25, (8, 8, 1)), (17, 33, (9, 7, 31)),
                                     (49, 3, (16, 16, 17)), (3, 5, (40, 41, 43)),
                                     (33, 1, (40, 41, 43))])
def test_pair_matrix(cuda, dtype, nx, ny, N):
    from gpawdft_b200 import blas
    import torch
    a = rand((nx,) + N, dtype, 1)
    b = rand((ny,) + N, dtype, 2)
    got = blas.pair_dots(torch.from_numpy(a).cuda(), nx,
                         torch.from_numpy(b).cuda(), ny)
    wide = complex if np.dtype(dtype).kind == 'c' else float
    a2, b2 = a.reshape(nx, -1).astype(wide), b.reshape(ny, -1).astype(wide)
    ref = a2.conj() @ b2.T
    n = a2.shape[1]
    bound = 4 * n * 2.0 ** -53 * (np.abs(a2) @ np.abs(b2).T)
    assert got.shape == ref.shape
    assert (np.abs(got - ref) <= 2 * bound).all()
    again = blas.pair_dots(torch.from_numpy(a).cuda(), nx,
                           torch.from_numpy(b).cuda(), ny)
    assert np.array_equal(got, again)


@pytest.mark.parametrize('dtype', [np.float64, np.complex128, np.float32,
                                   np.complex64])
@pytest.mark.parametrize('value', [np.inf, -np.inf, np.nan])
def test_not_finite(cuda, dtype, value):
    """An infinity or NaN in one vector reaches the pairs of that vector, with
    the sign it has there, and no other pair of its block."""
    from gpawdft_b200 import blas
    import torch
    a = rand((9, 6, 7, 8), dtype, 1)
    b = rand((11, 6, 7, 8), dtype, 2)
    a[4, 2, 3, 1] = value
    b[7, 5, 6, 7] = value
    got = blas.pair_dots(torch.from_numpy(a).cuda(), 9,
                         torch.from_numpy(b).cuda(), 11)
    cplx = np.dtype(dtype).kind == 'c'
    a, b = a.reshape(9, -1), b.reshape(11, -1)
    with np.errstate(invalid='ignore'):
        parts = [((a.real, b.real), (a.imag, b.imag)),
                 ((a.real, b.imag), (-a.imag, b.real))][:1 + cplx]
        ref = [sum(x.astype(float) @ y.astype(float).T
                   for x, y in (p if cplx else p[:1])) for p in parts]
    for g, r in zip((got.real, got.imag), ref):
        assert np.array_equal(np.isnan(g), np.isnan(r))
        assert np.array_equal(g[np.isinf(r)], r[np.isinf(r)])
        assert np.isfinite(g[np.isfinite(r)]).all()
