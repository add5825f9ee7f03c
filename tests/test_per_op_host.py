"""The host side of a per-op call: entry points resolved once, pointers and the
stream as plain integers."""

import ctypes
import threading

import pytest
import torch

from lbm_jax_autodiff_gb300 import _native as nat
from lbm_jax_autodiff_gb300 import _ops as op


class _Refused:
    def __enter__(self):
        raise AssertionError("a call of a loaded library takes no lock")

    def __exit__(self, *exc):
        return False


def test_a_call_neither_locks_nor_looks_up(monkeypatch):
    try:
        nat.load()
    except nat.NativeLibraryMissing:
        pytest.skip("the library is not built")
    k = ctypes.c_int()
    with monkeypatch.context() as m:
        m.setattr(nat, "_lock", _Refused())
        nat.call("lbm_plan_checkpoints", 100, 200, ctypes.byref(k))
    assert k.value == 100
    assert set(nat._functions) == set(nat.SIGNATURES)
    with pytest.raises(nat.LBMError):
        nat.call("lbm_plan_checkpoints", 100, 200, None)


def test_pointers_are_integers():
    t = torch.zeros(4)
    assert op.ptr(t) == t.data_ptr() and type(op.ptr(t)) is int and op.ptr(None) is None


@pytest.mark.gpu
def test_the_stream_is_the_callers(cuda):
    side = torch.cuda.Stream()
    seen = []

    def in_thread():
        with torch.cuda.stream(side):
            seen.append(op.stream())

    assert op.stream() == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(side):
        assert op.stream() == side.cuda_stream
    t = threading.Thread(target=in_thread)
    t.start()
    t.join()
    assert seen == [side.cuda_stream] and op.stream() != side.cuda_stream
