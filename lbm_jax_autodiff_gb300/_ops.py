"""Helpers shared by the per-op drop-in modules (core/*, geometry/*)."""

import torch

from . import _native as nat

FLAGS_EXACT = 1   # LBM_OP_EXACT_CONSTANTS


def dtype_code(t):
    if t.dtype == torch.float32:
        return nat.LBM_F32
    if t.dtype == torch.float64:
        return nat.LBM_F64
    raise TypeError("expected a float32 or float64 tensor, got %s" % t.dtype)


# Plain integers: ctypes converts them by the entry points' argument types.  A per-op
# call is bound by its host work (a step and its backward at 128x64x64 take the
# device 0.30 ms and took the host 1.28): torch.cuda.current_stream() alone is 3.1 us
# a call, the raw handle 0.2, and without it, a lock and a pointer object per
# argument the same step takes 0.94 ms.
def stream():
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def ptr(t):
    return None if t is None else t.data_ptr()


def cuda_contig(t, name):
    if not torch.is_tensor(t):
        raise TypeError("%s must be a torch tensor" % name)
    if not t.is_cuda:
        raise TypeError("%s must be on a CUDA device (this package has no CPU path)" % name)
    return t.contiguous()


def pop_dims(f):
    if f.dim() != 4 or f.shape[0] != 19:
        raise ValueError("populations must have shape (19, nx, ny, nz), got %s" % tuple(f.shape))
    return int(f.shape[1]), int(f.shape[2]), int(f.shape[3])


def call(name, *args):
    return nat.call(name, *args)
