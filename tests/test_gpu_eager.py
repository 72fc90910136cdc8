"""Eager calls served by C++ in one step (csrc/torch_shim/aten_shim.cpp): the same bits as the
operators behind them, and the calls they leave to those."""

import pytest
import torch
import torch.nn.functional as F

import kohaku_tt_b200 as ktt
from kohaku_tt_b200 import _lib
from tests.gpu_util import qkv

pytestmark = pytest.mark.gpu


def _both(monkeypatch, call):
    """call() by the C++ step and by the operators."""
    first = call()
    with monkeypatch.context() as m:
        m.setattr(_lib, "native", lambda: None)
        second = call()
    return first, second


def _with_grads(call, *leaves):
    leaves = [x.detach().requires_grad_() for x in leaves]
    out = call(*leaves)
    return (out, *torch.autograd.grad(out.float().square().sum(), leaves))


def _same(a, b):
    for x, y in zip(a, b, strict=True):
        assert x.shape == y.shape and torch.equal(x, y)


@pytest.mark.parametrize("kind", ["list", "cpu", "int64", "cuda"])
@pytest.mark.parametrize("sq,sk,d,causal", [(1, 300, 64, False), (1, 65, 128, False), (33, 129, 64, True)])
def test_lengths(cuda, monkeypatch, kind, sq, sk, d, causal):
    q, k, v = (x.to(cuda) for x in qkv(2, 4, 2, sq, sk, d, sq + sk))
    n = torch.tensor([sk, 1])
    lengths = {"list": n.tolist(), "cpu": n.int(), "int64": n, "cuda": n.int().to(cuda)}[kind]
    _same(*_both(monkeypatch, lambda: (ktt.sdpa(q, k, v, lengths, causal),)))
    _same(*_both(monkeypatch, lambda: _with_grads(lambda *x: ktt.sdpa(*x, lengths, causal), q, k, v)))


@pytest.mark.parametrize("kind", ["list", "cpu", "cuda"])
def test_packed(cuda, monkeypatch, kind):
    ktt.install()
    ends = torch.tensor([0, 1, 130, 300], dtype=torch.int32)
    cu = {"list": ends.tolist(), "cpu": ends, "cuda": ends.to(cuda)}[kind]
    q, k, v = (x[0].transpose(0, 1).contiguous().to(cuda) for x in qkv(1, 4, 2, 300, 300, 64, 3))
    call = lambda *x: ktt.sdpa_varlen(*x, cu, cu, is_causal=True)
    _same(*_both(monkeypatch, lambda: (call(q, k, v),)))
    _same(*_both(monkeypatch, lambda: _with_grads(call, q, k, v)))


@pytest.mark.parametrize("kind", ["list", "cpu"])
def test_packed_offsets_on_the_host_are_refused_in_a_capture(cuda, kind):
    # A replay would copy them from memory that is gone.
    ends = torch.tensor([0, 1, 130, 300], dtype=torch.int32)
    q, k, v = (x[0].transpose(0, 1).contiguous().to(cuda) for x in qkv(1, 4, 2, 300, 300, 64, 3))
    want = ktt.sdpa_varlen(q, k, v, ends, is_causal=True)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="capture"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            ktt.sdpa_varlen(q, k, v, ends.tolist() if kind == "list" else ends, is_causal=True)
    torch.cuda.synchronize()
    assert torch.equal(ktt.sdpa_varlen(q, k, v, ends, is_causal=True), want)


def test_decode_step(cuda, monkeypatch):
    q, k, v = (x.to(cuda) for x in qkv(3, 8, 2, 1, 200, 128, 4))
    kn, vn = k[:, :, :1] * 0.5, v[:, :, :1] * 0.5
    cos, sin = torch.randn(2, 200, 128, device=cuda).to(torch.bfloat16)
    lengths = torch.tensor([0, 127, 199], dtype=torch.int32, device=cuda)

    def call():
        kc, vc, after = k.clone(), v.clone(), torch.empty_like(lengths)
        return ktt.decode_step(q, kn, vn, kc, vc, lengths, cos, sin, lengths_out=after), kc, vc, after

    _same(*_both(monkeypatch, call))


def test_streams_and_what_the_step_leaves_alone(cuda):
    ktt.install()
    q, k, v = (x.to(cuda) for x in qkv(2, 8, 8, 300, 300, 64, 5))
    want = F.scaled_dot_product_attention(q, k, v)
    outs = []
    for _ in range(3):      # a workspace per stream: calls in flight on several do not meet
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            outs.append(F.scaled_dot_product_attention(q, k, v))
    torch.cuda.synchronize()
    for out in outs:
        assert torch.equal(out, want)
    # Other types and dropout stay torch's.
    f = F.scaled_dot_product_attention(q.float(), k.float(), v.float())
    assert f.dtype == torch.float32 and torch.allclose(f, want.float(), atol=2e-2)
    # A gradient of a gradient is an error.
    leaf = q.detach().requires_grad_()
    (dq,) = torch.autograd.grad(F.scaled_dot_product_attention(leaf, k, v).sum(), leaf, create_graph=True)
    with pytest.raises(RuntimeError, match="not differentiable"):
        dq.sum().backward()
