"""Which kernel a decode call takes, by its size: a cluster of CTAs per (batch, K / V head), or equal shares of all of
them, whose partials meet behind tickets; and the second of them in the forms that the first has taken over elsewhere."""

import os
import subprocess
import sys

import pytest
import torch

import kohaku_tt_b200 as ktt
from kohaku_tt_b200 import ops
from oracle import attention_oracle as ao
from tests import test_gpu_decode_step, test_zz_no_alloc
from tests.gpu_util import FWD_BOUND, qkv, rel
from tests.launched import launched

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


def _ranks(call, pairs, d, append=False):
    """CTAs of a pair's cluster in the one decode launch of `call`, 0 where the pairs are cut into equal shares."""
    (one,) = [k for k in launched(call) if "decode_kernel" in k.name]
    stages = {64: 6, 128: 3}[d]
    kind = f"decode_kernelILi{d}ELi{stages}ELb{int(append)}ELb"
    if kind + "1E" in one.name:
        assert one.grid == pairs * one.cluster
        return one.cluster
    assert kind + "0E" in one.name and one.cluster == 1
    return 0


# (pairs, keys the cache has room for, CTAs to a pair on 148 SMs). A tile is 64 keys; a rank has at most 1,024 keys, and
# beyond 512 as many times fewer as the clusters leave CTAs out of 296.
@pytest.mark.parametrize("pairs,sk,ranks", [
    (2, 64, 1), (2, 65, 2), (2, 129, 4), (2, 256, 4), (2, 257, 8), (2, 8192, 8), (2, 8193, 0), (24, 8192, 8),
    (40, 2048, 4), (40, 2214, 4), (40, 2215, 0), (56, 3099, 4), (56, 3100, 0), (80, 1107, 2), (80, 1108, 0),
    (148, 2048, 2), (148, 2049, 0), (160, 512, 1), (160, 645, 1), (160, 646, 0), (256, 1024, 1), (296, 1024, 1), (297, 64, 0),
])
@pytest.mark.parametrize("d", [64, 128])
def test_the_kernel_a_size_takes(cuda, pairs, sk, ranks, d):
    q = torch.zeros(pairs, 1, 1, d, dtype=torch.bfloat16, device=cuda)
    k = torch.zeros(pairs, 1, sk, d, dtype=torch.bfloat16, device=cuda)
    assert _ranks(lambda: ops.decode(q, k, k), pairs, d) == ranks


# Equal shares, which cut pairs between CTAs (few pairs) or end many of them in one (many).
@pytest.mark.parametrize("b,h,hk,smax,d,lengths", [
    (3, 16, 2, 8400, 128, [8399, 0, 4000]), (2, 14, 2, 9000, 64, [8191, 63]), (50, 4, 2, 3000, 64, None),
    (150, 2, 2, 300, 128, None), (150, 4, 2, 130, 64, None),
])
@pytest.mark.parametrize("by_position", [True, False])
def test_decode_step_on_shares(cuda, b, h, hk, smax, d, lengths, by_position):
    test_gpu_decode_step.test_decode_step_equals_the_three_ops(cuda, b, h, hk, smax, d, lengths, by_position)
    if by_position:
        q, new, cache = (torch.zeros(b, n, s, d, dtype=torch.bfloat16, device=cuda) for n, s in ((h, 1), (hk, 1), (hk, smax)))
        values = torch.zeros_like(cache)
        table, n = torch.zeros(smax, d, dtype=torch.bfloat16, device=cuda), torch.zeros(b, dtype=torch.int32, device=cuda)
        assert _ranks(lambda: ktt.decode_step(q, new, new, cache, values, n, table, table), b * hk, d, append=True) == 0


def test_calls_on_shares_have_one_scratch(cuda):
    """Tickets are back at zero and no call's partials reach another's counters or are read as its own."""
    shapes = [(2, 4, 2, 8300, 64), (80, 4, 2, 1500, 128), (3, 14, 2, 9000, 64), (80, 4, 2, 1500, 128), (300, 2, 1, 100, 64), (1, 16, 1, 8200, 128)]
    for i, (b, h, hk, smax, d) in enumerate(shapes):
        q, k, v = qkv(b, h, hk, 1, smax, d, 40 + i)
        lengths = torch.randint(1, smax + 1, (b,), generator=torch.Generator().manual_seed(i)).tolist()
        q_, k_, v_, n = q.to(cuda), k.to(cuda), v.to(cuda), torch.tensor(lengths, dtype=torch.int32, device=cuda)
        out, _ = ops.decode(q_, k_, v_, key_lengths=n)
        assert rel(out, ao.ruler_lengths(q, k, v, lengths)) <= FWD_BOUND, (i, b, h)
        assert _ranks(lambda: ops.decode(q_, k_, v_, key_lengths=n), b * hk, d) == 0


def test_static_calls_on_shares(cuda):
    # Large, then small over its stale partials, and another number of shares to a pair.
    for seed, shape, splits in ((1, (50, 4, 2, 128, 2200), 0), (2, (5, 8, 8, 64, 8200), 0), (3, (3, 16, 2, 128, 9000), 5), (4, (1, 16, 1, 128, 8300), 0)):
        static_out, regular_out, ruler = test_zz_no_alloc._both(cuda, seed, *shape, splits=splits)
        assert torch.equal(static_out, regular_out), seed
        assert rel(static_out, ruler) <= FWD_BOUND, seed


@pytest.mark.parametrize("splits", [1, 2, 3, 4, 5, 24, 0])   # shares of a pair, four to a round of the merge; 0: the most
def test_shares_keep_infinities(cuda, splits):
    n = 8200
    q, k, v = qkv(1, 16, 2, 1, n, 128, n)
    lengths = torch.tensor([n], dtype=torch.int32, device=cuda)
    ruler = ao.ruler_lengths(q, k, v, [n])
    v[0, :, 3, 5] = float("inf")
    v[0, :, n - 1, 7] = float("-inf")
    q, k, v = q.to(cuda), k.to(cuda), v.to(cuda)
    out = ops.decode(q, k, v, key_lengths=lengths, splits=splits)[0].cpu()
    assert (out[..., 5] == float("inf")).all() and (out[..., 7] == float("-inf")).all()
    rest = [c for c in range(128) if c not in (5, 7)]
    assert rel(out[..., rest], ruler[..., rest]) <= FWD_BOUND
    assert _ranks(lambda: ops.decode(q, k, v, key_lengths=lengths, splits=splits), 2, 128) == 0
