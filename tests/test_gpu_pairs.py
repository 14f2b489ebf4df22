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
