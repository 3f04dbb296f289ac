"""Decode steps and host-buffer calls against the oracle, in a process of its own so that a switch that the library reads once
per process (an environment variable) takes effect.  Run by tests/test_fattn_gpu.py::test_switches_read_once_per_process; prints
OK <max-abs> <rel-L2> per case."""
import sys

import numpy as np
import torch

sys.path.insert(0, __file__.rsplit("/tests/", 1)[0])
import crispasr_b200 as b200  # noqa: E402
from crispasr_b200 import abi  # noqa: E402
from oracle import oracle as orc  # noqa: E402
from tests.util import errors, gpu_op, randn_f16  # noqa: E402


def check(got, ref, name):
    e = errors(got, ref)
    assert e[0] <= 2e-3 and e[1] <= 1e-3, (name, e)
    print("OK", name, "%.2e %.2e" % e)


def main():
    rng = np.random.default_rng(77)
    # a Whisper decode step's cross-attention (one window: few units, many keys: splits), head_dim 64
    q, k, v = randn_f16(rng, (1, 6, 5, 64)), randn_f16(rng, (1, 6, 1500, 64)), randn_f16(rng, (1, 6, 1500, 64))
    check(gpu_op(b200, q, k, v, scale=0.125), orc.flash_attn_ext(q, k, v, scale=0.125), "cross")
    # a decoder step over a Q8_0 cache, ragged lengths
    lens = np.array([535, 500, 64, 1], np.int32)
    kq, vq = (orc.quantize_q8_0(rng.standard_normal((4, 8, 535, 128)).astype(np.float32)) for _ in "kv")
    q = randn_f16(rng, (4, 16, 1, 128))
    kw = dict(scale=128 ** -0.5, kv_type=abi.Q8_0, kv_len=lens)
    check(gpu_op(b200, q, kq, vq, **kw), orc.flash_attn_ext(q, kq, vq, **kw), "q8_0")
    # host buffers, pinned and pageable result
    q, k, v = (randn_f16(rng, (3, 4, 300, 64)) for _ in "qkv")
    args = [torch.from_numpy(x).pin_memory() for x in (q, k, v)]
    ref = orc.flash_attn_ext(q, k, v, scale=0.125)
    out = torch.empty((3, 300, 4, 64), dtype=torch.float32).pin_memory()
    check(b200.flash_attn_ext_host(*args, scale=0.125, out=out).numpy(), ref, "host, pinned")
    check(b200.flash_attn_ext_host(*args, scale=0.125).numpy(), ref, "host, pageable")
    assert b200.lib().b200_device_status() == 0


if __name__ == "__main__":
    main()
