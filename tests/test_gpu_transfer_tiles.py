"""The tile transfer kernels (gpw_transfer.cuh) on batches past the 8 MB up to
which complex K = 2 transfers are evaluated directly, every tap count and
element type, with tiles that are cut by the grid in both axes and chunks of
one and several planes: first and last member against the oracle
(c/bmgs/restrict.c, interpolate.c restated), bit-identical for float64 and
complex128."""
import numpy as np
import pytest

from helpers import TOL, oracle_dtype, rand, relerr
from oracle import layer as ol
from oracle.geometry import GridDescriptor as OGD, phase_cd_for_k

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nn', [1, 2, 3, 4])
@pytest.mark.parametrize('dtype', [np.complex128, np.complex64, np.float64,
                                   np.float32])
@pytest.mark.parametrize('N,pbc', [((10, 18, 34), 1), ((12, 21, 19), 0),
                                   ((9, 34, 16), (1, 0, 1))])
def test_batches_past_l2(cuda, N, pbc, dtype, nn):
    import torch
    from gpawdft_b200.grid_descriptor import GridDescriptor
    from gpawdft_b200.transformers import Transformer
    cell = tuple(0.25 * n for n in N)
    coarse, ocoarse = GridDescriptor(N, cell, pbc), OGD(N, cell, pbc)
    N2 = tuple(2 * n for n in N)
    fine, ofine = GridDescriptor(N2, cell, pbc), OGD(N2, cell, pbc)
    size = int(np.prod(fine.n_c)) * np.dtype(dtype).itemsize
    nin = 9 * 2 ** 20 // size + 1
    wide = oracle_dtype(dtype)
    ph = None
    if np.dtype(dtype).kind == 'c':
        ph = phase_cd_for_k(ofine, np.random.default_rng(3).uniform(-.5, .5,
                                                                    3))
    for gin, gout, ogin, ogout in ((fine, coarse, ofine, ocoarse),
                                   (coarse, fine, ocoarse, ofine)):
        a = torch.from_numpy(rand((nin,) + tuple(gin.n_c), dtype, 1)).cuda()
        got = Transformer(gin, gout, nn, dtype).apply(a, None, ph)
        op = ol.Transformer(ogin, ogout, nn, wide)
        for k in (0, nin - 1):
            ref = op.apply(a[k].cpu().numpy().astype(wide), None, ph)
            out = got[k].cpu().numpy()
            if np.dtype(dtype).itemsize == np.dtype(wide).itemsize:
                assert np.array_equal(out, ref), relerr(out, ref)
            else:
                assert relerr(out, ref) < TOL[np.dtype(dtype)]
