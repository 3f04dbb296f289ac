"""What the native call path takes and refuses as arguments (no GPU: a call that gets through ends at the missing device or
at a null cache)."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from crispasr_b200 import abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


@pytest.mark.parametrize("pos0", [3, 3.0, np.int64(3), torch.tensor(3)])
def test_append_positions_are_whatever_int_takes(b200, pos0):
    _append(b200, pos0=pos0)


def _host_call(b200, **kw):
    """A call on host tensors: returns, or ends at the missing device, once its arguments are converted."""
    x = torch.zeros(1, 1, 2, 64)
    try:
        b200.flash_attn_ext_host(x, x, x, **kw)
    except b200.B200Error as e:
        assert e.code in (abi.E_NO_DEVICE, abi.E_CUDA), e


class _Table:
    """An index table that is no tensor but knows its address."""

    def __init__(self):
        self.t = torch.ones(1, dtype=torch.int32)

    def data_ptr(self):
        return self.t.data_ptr()


@pytest.mark.parametrize("kw", [dict(scale="0.125"), dict(scale=torch.tensor(0.125)), dict(scale=np.float32(0.125)), dict(scale=1, n_past="2"),
                                dict(scale=1, n_past=1.0), dict(scale=1, causal=None, kv_len=None, kv_type=None, mask=None),
                                dict(scale=1, kv_len=np.ones(1, np.int32)), dict(scale=1, kv_len=_Table())])
def test_values_that_are_taken(b200, kw):
    """float() and int() of what is given, None where an argument may be left out, tables by address."""
    _host_call(b200, **kw)


@pytest.mark.parametrize("kw", [dict(scale=None), dict(scale=1, max_bias=None), dict(scale=1, softcap=None), dict(scale=1, n_past=None)])
def test_none_is_no_number(b200, kw):
    with pytest.raises(TypeError):
        _host_call(b200, **kw)


def test_scale_is_required(b200):
    with pytest.raises(KeyError):
        _host_call(b200)


def test_importing_the_package_imports_no_torch():
    """torch comes with the first use of a function that takes tensors, which is then the native one itself."""
    code = ("import sys, crispasr_b200 as b200\n"
            "from crispasr_b200 import abi, KvCache, SegmentScheduler\n"
            "assert 'torch' not in sys.modules\n"
            "f = b200.flash_attn_ext\n"
            "assert 'torch' in sys.modules and b200.flash_attn_ext is f is b200.op.flash_attn_ext and type(f).__name__ == 'builtin_function_or_method'\n"
            "from crispasr_b200 import flash_attn_ext_host\n"
            "try: b200.nothing\n"
            "except AttributeError: print('ok')\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr
