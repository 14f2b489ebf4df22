"""Reductions issued on two streams by one thread, and from a captured graph
between other calls: every call has scratch of its own, so the results are
those of calls made one after another, bit for bit."""
import numpy as np
import pytest

from helpers import rand

pytestmark = pytest.mark.gpu

# (vectors, vectors, points): large and small calls whose partial sums differ
# in number and place
SIZES = [(48, 48, 60000), (3, 5, 70000), (24, 25, 4096), (1, 1, 200000)]


def _calls(dtype):
    """Per size the three reductions of the library, as launches into a result
    tensor on the current stream."""
    import torch
    from gpawdft_b200 import _lib, arrays
    lib = _lib.load()
    for k, (nx, ny, n) in enumerate(SIZES):
        x = torch.from_numpy(rand((nx, n), dtype, 2 * k)).cuda()
        y = torch.from_numpy(rand((ny, n), dtype, 2 * k + 1)).cuda()
        code = arrays.code_of(x)

        def pairs(out, x=x, y=y, nx=nx, ny=ny, n=n):
            _lib.check(lib.gpw_dotc_pairs(code, nx, ny, n, arrays.ptr(x),
                                          arrays.ptr(y), arrays.ptr(out),
                                          arrays.stream()))

        def sums(out, x=x, nx=nx, n=n):
            _lib.check(lib.gpw_sum(code, nx, n, arrays.ptr(x),
                                   arrays.ptr(out), arrays.stream()))

        def dots(out, x=x, nx=nx, n=n):
            _lib.check(lib.gpw_dot(code, nx, n, arrays.ptr(x), arrays.ptr(x),
                                   arrays.ptr(out), arrays.stream()))
        for f, size in ((pairs, 2 * nx * ny), (sums, 2 * nx), (dots, nx)):
            yield f, lambda size=size: torch.zeros(size, dtype=torch.float64,
                                                   device='cuda')


@pytest.mark.parametrize('dtype', [np.float64, np.complex128])
def test_two_streams(cuda, dtype):
    import torch
    calls = list(_calls(dtype))
    want = []
    for f, new in calls:
        out = new()
        f(out)
        torch.cuda.synchronize()
        want.append(out.cpu())
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    jobs = [(i, streams[(i + r) % 2], calls[i][1]())
            for r in range(20) for i in range(len(calls))]
    torch.cuda.synchronize()
    for i, s, out in jobs:
        with torch.cuda.stream(s):
            calls[i][0](out)
    torch.cuda.synchronize()
    for i, s, out in jobs:
        assert torch.equal(out.cpu(), want[i]), i


def test_captured(cuda):
    import torch
    calls = list(_calls(np.complex128))
    outs = [new() for f, new in calls]
    want = []
    for (f, new), out in zip(calls, outs):
        f(out)
        torch.cuda.synchronize()
        want.append(out.cpu())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for (f, new), out in zip(calls, outs):
            f(out)
    other = torch.cuda.Stream()
    for _ in range(3):
        for out in outs:
            out.zero_()
        spare = [new() for f, new in calls]
        torch.cuda.synchronize()
        g.replay()
        with torch.cuda.stream(other):
            for (f, new), out in zip(calls, spare):
                f(out)
        torch.cuda.synchronize()
        for a, b, w in zip(outs, spare, want):
            assert torch.equal(a.cpu(), w) and torch.equal(b.cpu(), w)
