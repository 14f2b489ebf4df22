"""Device-array plumbing for the reference-facing API.

The reference's API works on NumPy arrays.  Here every call accepts either a
NumPy array (host; copied to the device, computed there, copied back -- the
end-to-end form) or a CUDA ``torch.Tensor`` (device-resident; zero copies).
PyTorch is used only for device memory and the current CUDA stream; all
arithmetic runs in libgpwgrid.so.
"""
import math

import numpy as np

try:
    import torch
except ImportError:  # pragma: no cover - torch is part of the image
    torch = None

from . import _lib

_NP_TO_CODE = {np.dtype(np.float64): _lib.GPW_F64,
               np.dtype(np.complex128): _lib.GPW_C128,
               np.dtype(np.float32): _lib.GPW_F32,
               np.dtype(np.complex64): _lib.GPW_C64}


if torch is not None:
    _TORCH_TO_NP = {torch.float64: np.dtype(np.float64),
                    torch.complex128: np.dtype(np.complex128),
                    torch.float32: np.dtype(np.float32),
                    torch.complex64: np.dtype(np.complex64)}
    _TORCH_TO_CODE = {t: _NP_TO_CODE[d] for t, d in _TORCH_TO_NP.items()}
    _NP_TO_TORCH = {d: t for t, d in _TORCH_TO_NP.items()}
    # the current stream's handle without a Stream object around it
    _raw_stream = getattr(torch._C, '_cuda_getCurrentRawStream', None)


def require_cuda():
    if torch is None or not torch.cuda.is_available():
        raise RuntimeError('gpawdft_b200 runs on a CUDA device (sm_100a); '
                           'no CPU fallback exists')
    _lib.load()


def is_device(a):
    return torch is not None and isinstance(a, torch.Tensor)


def stream():
    if _raw_stream is not None:
        return _raw_stream(torch.cuda.current_device())
    return torch.cuda.current_stream().cuda_stream


def code_of(a):
    if is_device(a):
        return _TORCH_TO_CODE[a.dtype]
    return _NP_TO_CODE[np.dtype(a.dtype)]


def np_dtype_of(a):
    if is_device(a):
        return _TORCH_TO_NP[a.dtype]
    return np.dtype(a.dtype)


def grids_of(a):
    """Number of grids in ``a`` (the product of its leading axes)."""
    return math.prod(a.shape[:-3])


def to_device(a):
    """CUDA tensor view of ``a`` (copied from the host for NumPy input)."""
    if is_device(a):
        if not a.is_cuda:
            require_cuda()
            raise ValueError('tensor must be on a CUDA device')
        if not a.is_contiguous():
            raise ValueError('array must be C-contiguous (as in the reference)')
        return a
    require_cuda()
    a = np.asarray(a)
    if not a.flags.c_contiguous:
        a = np.ascontiguousarray(a)
    if np.dtype(a.dtype) not in _NP_TO_TORCH:
        raise TypeError('unsupported dtype %s' % a.dtype)
    return torch.from_numpy(a).to('cuda', non_blocking=False)


def empty_like_device(shape, dtype):
    return torch.empty(tuple(shape), dtype=_NP_TO_TORCH[np.dtype(dtype)],
                       device='cuda')


def writeback(dst, src_dev):
    """Copy a device result into ``dst`` (NumPy) or nothing if it is ``dst``."""
    if is_device(dst):
        if dst.data_ptr() != src_dev.data_ptr():
            dst.copy_(src_dev)
        return
    dst[...] = src_dev.cpu().numpy().reshape(dst.shape)


def ptr(t):
    return t.data_ptr()


def phases_arg(phase_cd):
    """(3, 2) complex phase table -> 12 interleaved doubles (host), or None."""
    if phase_cd is None:
        return None, None
    p = np.ascontiguousarray(np.asarray(phase_cd, complex).reshape(3, 2))
    return p, p.__array_interface__['data'][0]
