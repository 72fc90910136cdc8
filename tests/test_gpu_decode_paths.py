"""Which kernel a decode call takes, by its size: a cluster of CTAs per (batch, K / V head), or equal shares of all of
them, whose partials meet behind tickets; and the second of them in the forms that the first has taken over elsewhere."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# A process of its own: set-up is once per process and device.
SETUP = """
import ctypes, torch
from kohaku_tt_b200 import _lib
lib, dev = _lib.lib(), torch.device("cuda:0")

def call(entry, b, hk, sk, d):
    q, k = torch.randn(b, 2 * hk, 1, d, device=dev).bfloat16(), torch.randn(b, hk, sk, d, device=dev).bfloat16()
    out, a = torch.empty_like(q), _lib.DecodeArgs()
    a.batch, a.heads, a.kv_heads, a.sq, a.sk, a.d, a.dv, a.scale = b, 2 * hk, hk, 1, sk, d, d, d ** -0.5
    a.q, a.k, a.v, a.out = q.data_ptr(), k.data_ptr(), k.data_ptr(), out.data_ptr()
    for name, t in (("q_strides", q), ("k_strides", k), ("v_strides", k), ("out_strides", out)):
        for i in range(3):
            getattr(a, name)[i] = t.stride(i)
    if entry == "ktt_b200_decode":
        a.scratch_bytes = lib.ktt_b200_decode_scratch_bytes(ctypes.byref(a))
        scratch = torch.zeros(a.scratch_bytes, dtype=torch.uint8, device=dev)
        a.scratch = scratch.data_ptr()
    _lib.check(getattr(lib, entry)(ctypes.byref(a), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), entry)
    torch.cuda.synchronize()
    return _lib.counters()["kernel_setups"]

first = call(%r, 1, 2, 64, 64)
for b, hk, sk, d in %r:
    assert call(%r, b, hk, sk, d) == first, (b, hk, sk, d)
"""

# Clusters of 1, 2, 4 and 8, and shares (more than 1,024 keys to a rank, more pairs than CTAs).
SIZES = [(1, 2, 300, 64), (40, 1, 300, 64), (100, 1, 300, 64), (200, 1, 300, 64), (2, 2, 9000, 64), (300, 1, 64, 64)]


@pytest.mark.parametrize("entry,sizes", [
    ("ktt_b200_decode", SIZES),
    ("ktt_b200_decode_static", SIZES + [(b, hk, sk, 128) for b, hk, sk, _ in SIZES if b * hk <= 207]),
])
def test_the_first_call_sets_up_calls_of_every_size(cuda, entry, sizes):
    subprocess.run([sys.executable, "-c", SETUP % (entry, sizes, entry)], cwd=ROOT, check=True)
