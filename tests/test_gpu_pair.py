"""The forward kernel of two query tiles per CTA (csrc/fwd_pair.cu): head dims it zero-fills and
masks with a row per query, at the edges of its tiles, against the float64 ruler."""

import ctypes
import math

import pytest
import torch
import torch.nn.functional as F

import kohaku_tt_b200 as ktt
from kohaku_tt_b200 import _lib, ops
from oracle import attention_oracle as ao
from tests.gpu_util import FWD_BOUND, LSE_RMS, qkv, rel, rms

pytestmark = pytest.mark.gpu


def _check(cuda, q, k, v, mask=None, causal=False, lengths=None, kernel="flash_pair", counted="attention_flash"):
    before = ktt.counters()[counted]
    ln = None if lengths is None else torch.tensor(lengths, dtype=torch.int32, device=cuda)
    out, lse = ops.sdpa_forward(q.to(cuda), k.to(cuda), v.to(cuda), causal=causal, key_lengths=ln,
                                mask=None if mask is None else mask.to(cuda), kernel=kernel)
    torch.cuda.synchronize()
    _lib.device_status()
    assert ktt.counters()[counted] == before + 1   # the kernel that was meant took it
    if lengths is not None:
        ruler = ao.ruler_lengths(q, k, v, lengths)
    else:
        ruler = ao.ruler_dense(q, k, v, mask=mask, causal=causal)
        assert rms(lse, ao.ruler_lse(q, k, v, mask=mask, causal=causal)) <= LSE_RMS
    assert rel(out, ruler) <= FWD_BOUND


# One key or row past a tile, a tile exactly, one short of it; a block with 1, 16, 17 and 128 keys;
# one tile (its keys in two halves), an odd number of tiles, more tiles than CTAs.
@pytest.mark.parametrize("b,h,hk,sq,sk,d,dv,causal", [
    (1, 1, 1, 1, 1, 8, 8, False), (1, 2, 1, 128, 144, 80, 80, False), (2, 3, 3, 129, 257, 80, 80, False),
    (1, 6, 2, 127, 145, 96, 96, True), (2, 2, 2, 300, 128, 40, 40, True), (1, 5, 1, 400, 400, 72, 72, True),
    (1, 4, 2, 130, 200, 64, 128, False), (1, 2, 2, 200, 130, 120, 16, False), (40, 8, 8, 257, 257, 88, 88, False),
])
def test_head_dims(cuda, b, h, hk, sq, sk, d, dv, causal):
    _check(cuda, *qkv(b, h, hk, sq, sk, d, sq + sk + d, dv=dv), causal=causal)


# The tiles of a CTA take turns from five blocks of keys on: both sides of that line, tiles of unequal
# length and items in which the second tile has no block or is not there.
@pytest.mark.parametrize("b,h,hk,sq,sk,d,causal,lengths", [
    (2, 75, 75, 256, 512, 80, False, None), (2, 75, 75, 256, 513, 80, False, None), (1, 101, 101, 257, 700, 96, True, None),
    (1, 30, 10, 700, 640, 72, True, None), (3, 50, 50, 129, 1100, 128, False, [1100, 1, 515]), (2, 40, 20, 520, 900, 120, True, [900, 130]),
])
def test_turns(cuda, b, h, hk, sq, sk, d, causal, lengths):
    q, k, v = qkv(b, h, hk, sq, sk, d, sq + sk + d)
    if lengths is not None and causal:   # (the ruler for lengths is not causal: the plain one on each sequence)
        out, _ = ops.sdpa_forward(q.to(cuda), k.to(cuda), v.to(cuda), causal=True, kernel="flash_pair",
                                  key_lengths=torch.tensor(lengths, dtype=torch.int32, device=cuda))
        for i, n in enumerate(lengths):
            one = ao.ruler_dense(q[i:i + 1], k[i:i + 1, :, :n], v[i:i + 1, :, :n], causal=True)
            assert rel(out[i:i + 1], one) <= FWD_BOUND
        return
    _check(cuda, q, k, v, causal=causal, lengths=lengths)


# Calls that other kernels take too: just inside and outside the rounds, tiles and keys between them.
@pytest.mark.parametrize("h,sq,sk,d,masked", [
    (37, 512, 96, 64, True), (38, 400, 77, 64, True), (148, 256, 40, 64, False), (50, 300, 320, 64, True),
    (75, 130, 321, 64, True), (38, 512, 321, 64, False), (149, 256, 33, 128, True), (80, 256, 97, 128, False),
    (80, 200, 129, 128, True), (112, 512, 64, 128, False),
])
def test_few_keys(cuda, h, sq, sk, d, masked):
    q, k, v = qkv(1, h, h, sq, sk, d, h + sq + sk)
    keep = torch.rand(1, 1, 1, sk, generator=torch.Generator().manual_seed(h)) > 0.3
    keep[..., 0] = True
    _check(cuda, q, k, v, mask=keep if masked else None, kernel="auto")


# Pairs beyond whole rounds of one per SM run as halves: both sides of that line (148 and 149, 222 and 223 pairs), of two
# and of more rounds, tiles without a partner, two to six blocks of keys (an odd number shares unevenly), a last block
# of one key, and a mask that leaves a half without a visible key.
@pytest.mark.parametrize("b,h,hk,sq,sk,d,masked", [
    (1, 148, 148, 256, 129, 64, False), (1, 149, 149, 256, 129, 64, False), (2, 75, 75, 200, 144, 80, False),
    (1, 222, 222, 129, 300, 40, False), (1, 223, 223, 129, 300, 40, False), (2, 35, 35, 600, 257, 80, False),
    (1, 160, 20, 130, 700, 128, False), (5, 30, 30, 256, 513, 96, False), (1, 302, 302, 256, 384, 64, False),
    (2, 75, 75, 256, 320, 64, True), (1, 150, 150, 150, 290, 128, True), (2, 35, 7, 600, 260, 64, True),
])
def test_last_round_in_halves(cuda, b, h, hk, sq, sk, d, masked):
    q, k, v = qkv(b, h, hk, sq, sk, d, h + sq + sk)
    keep = None
    if masked:
        keep = torch.rand(b, 1, 1, sk, generator=torch.Generator().manual_seed(h)) > 0.3
        keep[..., 0] = True
        keep[0, ..., 128:] = False
    _check(cuda, q, k, v, mask=keep)


# One row behind the last whole tile goes without a tile: both sides of the lines (148 and 150 tiles, one round of pairs
# and more, a last round of 74 and 75), keys short of, at and past a warp's 32 and a pass of 256, groups of heads, lengths.
@pytest.mark.parametrize("b,h,hk,sq,sk,d,dv,lengths", [
    (1, 74, 74, 257, 257, 80, 80, None), (1, 75, 75, 257, 257, 80, 80, None), (2, 74, 74, 257, 32, 64, 64, None), (1, 149, 149, 257, 33, 40, 40, None),
    (2, 111, 111, 257, 256, 64, 128, None), (1, 223, 223, 257, 1152, 96, 96, None), (1, 223, 223, 257, 1153, 8, 8, None),
    (2, 80, 40, 129, 31, 120, 24, None), (1, 160, 10, 129, 700, 128, 128, None), (3, 60, 60, 257, 300, 72, 72, [1, 300, 130]),
])
def test_last_row_apart(cuda, b, h, hk, sq, sk, d, dv, lengths):
    q, k, v = qkv(b, h, hk, sq, sk, d, h + sq + sk, dv=dv)
    _check(cuda, q, k, v, lengths=lengths)
    # (One row in 257 hardly shows in the whole's error.)
    ln = None if lengths is None else torch.tensor(lengths, dtype=torch.int32, device=cuda)
    out, _ = ops.sdpa_forward(q.to(cuda), k.to(cuda), v.to(cuda), key_lengths=ln, kernel="flash_pair")
    last = q[:, :, -1:]
    assert rel(out[:, :, -1:], ao.ruler_dense(last, k, v) if lengths is None else ao.ruler_lengths(last, k, v, lengths)) <= FWD_BOUND


# Dense calls without a mask take the kernel whose rounds are the better filled: both sides of that line, causal and
# not, one and several tiles per item, an odd number of (tile, head)s, lengths that are no multiple of a tile.
@pytest.mark.parametrize("b,h,hk,sq,sk,d,causal", [
    (8, 14, 2, 256, 256, 64, True), (1, 14, 2, 1024, 1024, 64, True), (3, 15, 3, 500, 500, 64, True), (9, 9, 3, 385, 385, 64, True),
    (2, 12, 12, 700, 700, 64, False), (2, 20, 20, 300, 900, 64, False), (8, 16, 16, 200, 200, 128, True), (2, 5, 1, 400, 250, 128, True),
])
def test_better_filled_rounds(cuda, b, h, hk, sq, sk, d, causal):
    _check(cuda, *qkv(b, h, hk, sq, sk, d, b + sq + sk + d), causal=causal, kernel="auto")


# Few rows: the warp-MMA kernel, up to where the tiles fill (both sides of the line).
@pytest.mark.parametrize("b,h,sq,sk,d,kind,kernel", [
    (1, 1, 1, 1, 8, None, "mma"), (2, 16, 49, 49, 32, None, "mma"), (64, 16, 64, 64, 32, "bf16", "mma"),
    (8, 16, 128, 128, 64, "values", "mma"), (2, 16, 16, 16, 80, None, "mma"), (1, 16, 64, 64, 64, "random", "mma"),
    (2, 16, 144, 144, 32, None, "flash"), (2, 16, 128, 128, 80, None, "flash"), (8, 16, 197, 197, 64, "random", "flash"),
])
def test_few_rows(cuda, b, h, sq, sk, d, kind, kernel):
    q, k, v = qkv(b, h, h, sq, sk, d, sq + sk + d)
    _check(cuda, q, k, v, mask=_mask(kind, b, h, sq, sk) if kind else None, kernel="auto", counted="attention_" + kernel)


def test_head_dim_80_with_key_lengths_and_a_key_mask(cuda):
    q, k, v = qkv(3, 4, 2, 200, 300, 80, 5)
    _check(cuda, q, k, v, lengths=[300, 1, 130])
    keep = torch.rand(3, 1, 1, 300, generator=torch.Generator().manual_seed(6)) > 0.3
    keep[..., 0] = True
    _check(cuda, q, k, v, mask=keep)


def _mask(kind, b, h, sq, sk):
    g = torch.Generator().manual_seed(sq + sk)
    if kind == "values":                       # every piece has values
        return torch.randn(b, h, sq, sk, generator=g)
    if kind == "bf16":
        return torch.randn(b, 1, sq, sk, generator=g).to(torch.bfloat16)
    if kind == "fp16":
        return torch.randn(1, h, sq, sk, generator=g).to(torch.float16)
    if kind == "random":                       # yes / no everywhere
        keep = torch.rand(b, 1, sq, sk, generator=g) > 0.5
        keep[..., 0] = True
        return keep
    keep = torch.ones(sq, sk, dtype=torch.bool).tril(max(sk - sq, 0))   # blocks hidden, free and mixed
    if kind == "causal":
        return keep
    add = torch.zeros(1, 1, sq, sk).masked_fill(~keep, -math.inf)
    if kind == "mixed":                        # a value in one piece, and a row that sees nothing
        add[..., 5, 3] = -1.5
        add[..., sq // 2, :] = -5e5
    return add


@pytest.mark.parametrize("kind", ["values", "bf16", "fp16", "random", "causal", "additive", "mixed"])
@pytest.mark.parametrize("b,h,hk,sq,sk,d", [
    (2, 4, 4, 257, 300, 64), (1, 6, 2, 128, 129, 128), (2, 2, 2, 33, 520, 96), (2, 16, 16, 700, 700, 64),
])
def test_masks_with_a_row_per_query(cuda, kind, b, h, hk, sq, sk, d):
    q, k, v = qkv(b, h, hk, sq, sk, d, sq + sk + d)
    _check(cuda, q, k, v, mask=_mask(kind, b, h, sq, sk))


def test_mask_strides(cuda):
    # A slice of a wider mask (rows start anywhere), a mask broadcast over the keys, an odd width.
    q, k, v = qkv(2, 4, 4, 150, 203, 64, 9)
    wide = torch.randn(2, 1, 150, 211, generator=torch.Generator().manual_seed(7)).to(torch.bfloat16)
    _check(cuda, q, k, v, mask=wide[..., 5:208])
    _check(cuda, q, k, v, mask=wide[..., :1])


# A last block of 1 to 16 keys past a multiple of 32: the columns up to the next multiple belong to no
# product of 16, and hold what the kernel before left in tensor memory.
@pytest.mark.parametrize("d", [64, 80, 128])
@pytest.mark.parametrize("sk", [1, 16, 77, 129, 240])
def test_a_key_mask_reads_only_what_the_call_computed(cuda, sk, d):
    g = torch.Generator().manual_seed(sk)
    q, k, v = (x.to(cuda) for x in qkv(2, 37, 37, 500, sk, d, sk + d))
    keep = torch.rand(2, 1, 1, sk, generator=g) > 0.3
    keep[..., 0] = True
    keep = keep.to(cuda)
    # Every score of every SM's two tiles a NaN, and P over them where it shares their columns.
    poison = [x.to(cuda) for x in qkv(1, 148, 148, 256, 128, 80, 1)]
    poison[1][:] = math.nan
    want, want_lse = ops.sdpa_forward(q, k, v, mask=keep, kernel="flash_pair")
    assert rel(want, ao.ruler_dense(q.cpu(), k.cpu(), v.cpu(), mask=keep.cpu())) <= FWD_BOUND
    for _ in range(3):
        ops.sdpa_forward(*poison, kernel="flash_pair")
        out, lse = ops.sdpa_forward(q, k, v, mask=keep, kernel="flash_pair")
        assert torch.equal(out, want) and torch.equal(lse, want_lse)


def test_more_mask_planes_than_a_grid_dimension(cuda):
    # A mask of its own for each of 4,096 x 16 (batch, head) pairs (windows of a bitmap, one key apart).
    g = torch.Generator(cuda).manual_seed(8)
    q, k, v = (torch.randn(4096, 16, 200, 80, device=cuda, dtype=torch.bfloat16, generator=g) for _ in range(3))
    bits = torch.rand(4096 + 16 * 4096 + 200 * 200, device=cuda, generator=g) > 0.4
    mask = bits.as_strided((4096, 16, 200, 200), (1, 4096, 200, 1))
    out, _ = ops.sdpa_forward(q, k, v, mask=mask, kernel="flash_pair")
    for b, h in ((0, 0), (2047, 15), (4095, 0), (4095, 14), (4095, 15)):
        part = [x[b:b + 1, h:h + 1].cpu() for x in (q, k, v, mask)]
        assert rel(out[b:b + 1, h:h + 1], ao.ruler_dense(*part[:3], mask=part[3])) <= FWD_BOUND


# The plan of a mask a part of the call at a time: batch entries, K / V heads, heads of one, query rows
# (the last of them a single one).
@pytest.mark.parametrize("b,h,hk,sq,kind,parts", [
    (3, 6, 2, 300, "values", 2), (3, 6, 2, 300, "values", 5), (3, 6, 2, 300, "values", 12), (3, 6, 2, 300, "values", 40),
    (2, 4, 2, 257, "bf16", 4), (1, 4, 4, 257, "fp16", 8), (2, 2, 1, 257, "additive", 2), (2, 2, 1, 257, "causal", 2),
])
def test_parts_of_a_plan(cuda, monkeypatch, b, h, hk, sq, kind, parts):
    sizes = []

    def workspace(args, device):
        whole = _lib.lib().ktt_b200_sdpa_forward_workspace(ctypes.byref(args))
        buf = torch.empty(256 + (whole - 256) // parts, dtype=torch.uint8, device=device)
        sizes.append(buf.numel())
        args.workspace, args.workspace_bytes = buf.data_ptr(), buf.numel()
        return buf

    monkeypatch.setattr(ops, "forward_workspace", workspace)
    operands = qkv(b, h, hk, sq, 200, 64, sq + parts)
    _check(cuda, *operands, mask=_mask(kind, b, h, sq, 200))
    # Head views of [B, S, H * D], a mask whose rows are a slice of wider ones.
    views = [x.transpose(1, 2).contiguous().transpose(1, 2) for x in operands]
    _check(cuda, *views, mask=_mask(kind, b, h, sq, 211)[..., :200])
    assert len(sizes) == 2


def test_a_plan_takes_bounded_memory(cuda):
    # 1.8 GB if it were whole; and none where the device has no room for it. (No cached segment is left
    # that has room beside a tensor of this test.)
    torch.cuda.empty_cache()
    g = torch.Generator(cuda).manual_seed(3)
    q, k, v = (torch.randn(128, 16, 400, 80, device=cuda, dtype=torch.bfloat16, generator=g) for _ in range(3))
    bits = torch.randn(128 + 16 * 128 + 400 * 400, device=cuda, generator=g)
    mask = bits.as_strided((128, 16, 400, 400), (1, 128, 400, 1))
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    counts = ktt.counters()
    out, lse = ops.sdpa_forward(q, k, v, mask=mask)
    assert ktt.counters()["attention_flash"] == counts["attention_flash"] + 1
    results = out.numel() * 2 + lse.numel() * 4
    assert torch.cuda.max_memory_allocated() - before <= results + (1025 << 20)
    for b, h in ((0, 0), (63, 7), (127, 15)):
        part = [x[b:b + 1, h:h + 1].cpu() for x in (q, k, v, mask)]
        assert rel(out[b:b + 1, h:h + 1], ao.ruler_dense(*part[:3], mask=part[3])) <= FWD_BOUND
    for call in (lambda: ops.sdpa_forward(q, k, v, mask=mask)[0], lambda: F.scaled_dot_product_attention(q, k, v, attn_mask=mask)):
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(cuda).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + results + (64 << 20)) / total)
        counts = ktt.counters()
        try:
            again = call()
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        assert ktt.counters()["attention_mma"] == counts["attention_mma"] + 1
        assert rel(again, out.cpu()) <= FWD_BOUND
        del again
