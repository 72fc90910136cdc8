"""Calls of head dim 64 and 128 that more than one tcgen05 kernel takes: what a caller hands over means the same to each."""

import ctypes

import pytest
import torch

from kohaku_tt_b200 import _lib, ops
from tests.gpu_util import qkv
from tests.launched import launched

pytestmark = pytest.mark.gpu


def _forward(q, k, v, causal, workspace=None):
    args, keep = ops._dense_args(q, k, v, None, None, causal, None, "auto")
    out = torch.full_like(q, float("nan"))
    args.out = out.data_ptr()
    ops._set3(args.out_strides, out.stride()[:3])
    if workspace is not None:
        args.workspace, args.workspace_bytes = workspace.data_ptr(), workspace.numel()
    _lib.check(_lib.lib().ktt_b200_sdpa_forward(ctypes.byref(args), ops._stream(q.device)), "sdpa_forward")
    return out


# More items than two per SM, so that they are drawn from a counter. `fill`: what the workspace holds before the first
# call, `again`: before every other (None: as it was left).
@pytest.mark.parametrize("b,h,hk,n,d,at,size,fill,again", [
    (4, 20, 20, 1000, 64, 0, 256, 0, None), (4, 20, 20, 1000, 64, 4, 256, 0, None), (4, 20, 20, 1000, 64, 0, 64, 1, None), (4, 20, 20, 1000, 64, 8, 16, 0, None),
    (5, 32, 8, 640, 128, 0, 256, 0, None), (5, 32, 8, 640, 128, 4, 256, 0, None), (5, 32, 8, 640, 128, 4, 16, 0, 0), (5, 32, 8, 640, 80, 4, 256, 0, None),
])
def test_a_workspace_of_any_size_and_alignment(cuda, b, h, hk, n, d, at, size, fill, again):
    q, k, v = (t.to(cuda) for t in qkv(b, h, hk, n, n, d, n + d))
    assert any("fwd_pair" in x.name for x in launched(lambda: _forward(q, k, v, True)))
    want = _forward(q, k, v, True)   # (none: a fixed deal of the same items)
    workspace = torch.full((at + size + 64,), fill, dtype=torch.uint8, device=cuda)
    for _ in range(3):
        assert torch.equal(_forward(q, k, v, True, workspace[at:at + size]), want)
        if again is not None:
            workspace.fill_(again)
    assert (workspace[at + size:] == fill).all()


# Halves of a last round, dealt and drawn (344 items for 148 SMs).
def test_halves_from_a_counter_and_from_a_fixed_deal(cuda):
    q, k, v = (t.to(cuda) for t in qkv(1, 20, 20, 4096, 4096, 64, 5))
    workspace = torch.zeros(256, dtype=torch.uint8, device=cuda)
    drawn = [_forward(q, k, v, False, workspace) for _ in range(2)]
    dealt = _forward(q, k, v, False)
    assert torch.equal(drawn[0], dealt) and torch.equal(drawn[1], dealt) and dealt.isfinite().all()


# A trace and a dump are written by the kernels that took these calls before this one did.
@pytest.mark.parametrize("b,h,hk,n,sk,d,causal,kernel", [
    (4, 20, 20, 1000, 1000, 64, True, "fwd_row"), (2, 10, 10, 4096, 77, 64, False, "fwd_row"), (5, 32, 8, 640, 640, 128, True, "fwd_tc5"),
])
def test_what_is_traced_stays_with_the_traced_kernels(cuda, b, h, hk, n, sk, d, causal, kernel):
    q, k, v = (t.to(cuda) for t in qkv(b, h, hk, n, sk, d, n + d))
    handle = _lib.lib()
    call = lambda: _forward(q, k, v, causal)
    assert any("fwd_pair" in x.name for x in launched(call))
    trace = torch.zeros((64 + 1024) * 8, dtype=torch.int64, device=cuda)
    handle.ktt_b200_set_trace(trace.data_ptr())
    try:
        assert any(kernel in x.name for x in launched(call))
    finally:
        handle.ktt_b200_set_trace(None)
    torch.cuda.synchronize()
    assert trace[64 * 8] > 0   # the first CTA's start
    if d == 64:
        blocks = (sk + 127) // 128
        dump = torch.full((blocks * (2 * 128 * 128 + 2 * 128) + 128 * 64 + 2 * 128,), float("nan"), device=cuda)
        assert handle.ktt_b200_set_dump(dump.data_ptr(), b - 1, h - 1, 1, blocks) == 0
        try:
            assert any(kernel in x.name for x in launched(call))
        finally:
            handle.ktt_b200_set_dump(None, 0, 0, 0, 0)
        torch.cuda.synchronize()
        assert dump[-256:].isfinite().all()   # the tile's last maxima and sums
    assert any("fwd_pair" in x.name for x in launched(call))
    _lib.device_status()


# On 148 SMs. One round of tiles stays with the kernel of whole tiles; beyond it the kernel whose rounds are better filled
# takes the call. `kind`: of the paired kernel, turns (head dim 128, five blocks of keys on) and a last round in halves.
@pytest.mark.parametrize("b,h,hk,n,d,causal,kernel,kind", [
    (8, 14, 2, 512, 64, True, "pair", "00"), (2, 32, 8, 1024, 64, True, "pair", "00"), (4, 20, 20, 200, 64, True, "pair", "00"),
    (1, 20, 20, 1024, 64, False, "pair", "00"), (1, 20, 20, 4096, 64, False, "pair", "01"), (2, 20, 20, 1000, 64, False, "pair", "01"),
    (8, 16, 16, 200, 128, True, "pair", "00"), (8, 14, 2, 640, 128, True, "pair", "10"), (3, 24, 24, 257, 128, False, "pair", "00"),
    (1, 14, 2, 1024, 64, True, "row", ""), (1, 14, 2, 2048, 64, True, "row", ""), (4, 20, 20, 257, 64, True, "row", ""),
    (4, 20, 20, 640, 64, False, "row", ""), (8, 14, 2, 1000, 64, True, "row", ""), (1, 37, 37, 512, 64, True, "row", ""),
    (1, 20, 20, 1024, 128, False, "tc5", ""), (3, 24, 24, 513, 128, False, "tc5", ""), (2, 20, 20, 1024, 128, True, "tc5", ""),
    (3, 24, 24, 384, 128, True, "tc5", ""), (1, 37, 37, 512, 128, True, "tc5", ""),
])
def test_the_kernel_a_call_takes(cuda, b, h, hk, n, d, causal, kernel, kind):
    q = torch.zeros(b, h, n, d, dtype=torch.bfloat16, device=cuda)
    k = torch.zeros(b, hk, n, d, dtype=torch.bfloat16, device=cuda)
    (one,) = [x for x in launched(lambda: _forward(q, k, k, causal)) if "fwd_" in x.name]
    assert f"fwd_{kernel}_kernel" in one.name
    if kind:
        assert f"fwd_pair_kernelILi{d}ELi0ELb{kind[0]}ELb{kind[1]}E" in one.name
