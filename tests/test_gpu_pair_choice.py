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
