"""What the native call path takes and refuses as arguments (no GPU: a call that gets through ends at the missing device or
at a null cache)."""
import ctypes as C

import numpy as np
import pytest
import torch

from crispasr_b200 import abi


def _append(b200, stream=0, pos=None, pos0=0):
    """kv_append on a null cache: every argument is converted first."""
    x = torch.zeros(1, 1, 1, 64)
    with pytest.raises(b200.B200Error) as e:
        b200.op._kv_append(0, 0, x, x, pos, pos0, stream)
    assert e.value.code == abi.E_NULL


class _Stream:
    def __init__(self, v):
        self._as_parameter_ = v


@pytest.mark.parametrize("stream", [0, 4096, C.c_void_p(4096), C.c_void_p(), _Stream(C.c_void_p(4096)), _Stream(4096)])
def test_streams_that_are_taken(b200, stream):
    """Integers, ctypes pointers, and whatever ctypes itself would take as a pointer (torch.cuda.Stream)."""
    _append(b200, stream=stream)


@pytest.mark.parametrize("stream", ["default", 1.5, _Stream("default")])
def test_streams_that_are_refused(b200, stream):
    x = torch.zeros(1, 1, 1, 64)
    with pytest.raises((TypeError, AttributeError)):
        b200.op._kv_append(0, 0, x, x, None, 0, stream)


def test_append_refuses_host_rows_and_host_positions(b200):
    """Rows in host memory on the default stream, and positions that are no tensor, never reach the kernel."""
    x = torch.zeros(1, 1, 1, 64)
    with pytest.raises(ValueError):
        b200.op._kv_append(0, 0, x, x, None, 0, None)
    with pytest.raises(TypeError):
        b200.op._kv_append(0, 0, x, x, np.zeros(1, np.int32), 0, 0)
    _append(b200, pos=torch.zeros(1, dtype=torch.int32))
