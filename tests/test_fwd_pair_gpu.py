"""The forward kernel for grids that fill the chip (two query tiles per CTA, persistent) against the fp32 composite: even and
odd numbers of query tiles, key counts around the key step, every mask kind, and packed batches with empty
sequences, sequences past the stated maximum and rows outside all sequences.  Tolerances: helpers.assert_close."""
import pytest
import torch

import mha_manual  # noqa: F401  registers torch.ops.mha_manual.*
from nvfuserexamples_b200 import api, capi
from oracle import composite
from tests import helpers
from tests.test_fwd_rules import pair_pays

pytestmark = pytest.mark.gpu


def inputs(B, H, S_q, S_k, D, dtype, seed, dev):
    g = torch.Generator(device=dev).manual_seed(seed)
    r = lambda S: torch.randn(B, H, S, D, device=dev, generator=g).to(dtype)
    return r(S_q), r(S_k), r(S_k)


def takes_pairs(B, H, S_q, S_k, lengths=True, packed_rows=0):   # the library's rule, so that the sizes below keep to it
    return pair_pays(torch.cuda.get_device_properties(0).multi_processor_count, B, H, S_q, S_k, packed_rows, lengths)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("mask", ["none", "seqlen", "key", "key_inf"])
@pytest.mark.parametrize("B,H,S_q,S_k", [(37, 4, 129, 257), (19, 8, 256, 384), (12, 16, 600, 385), (8, 8, 640, 511), (19, 8, 200, 900)])
def test_pair_kernel_matches_the_composite(cuda_device, B, H, S_q, S_k, mask, dtype):
    D = 128
    assert takes_pairs(B, H, S_q, S_k)
    q, k, v = inputs(B, H, S_q, S_k, D, dtype, S_q + S_k, cuda_device)
    lens = (torch.arange(B, device=cuda_device, dtype=torch.int32) * 7919) % S_k + 1
    kw, add = {}, None
    if mask == "seqlen":
        kw["seqlens"], add = lens, composite.padding_add_mask(lens, S_k)
    elif mask != "none":   # -inf on the padded keys; the first key of every third batch element as well
        add = composite.padding_add_mask(lens, S_k, -10000.0 if mask == "key" else float("-inf"))
        if mask == "key_inf" and S_k > 1:
            add[::3, ..., 0] = torch.where(lens[::3] > 1, float("-inf"), 0.0).reshape(-1, 1, 1)
        kw["mask"] = add.reshape(B, S_k)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    o, lse = api.fmha_forward(q, k, v, status=status, **kw)
    assert capi.check_status(status) == [0, 0, 0, 0]
    ref = composite.attention_fp32(q, k, v, add_mask=add)
    # Short sums (valid lengths go down to one key) break the elementwise bar with bf16 (helpers.assert_close): there no further
    # off than twice the 16-bit composite.
    if dtype == torch.bfloat16:
        sc = torch.matmul(q, k.transpose(-1, -2)) * D ** -0.5
        eager = torch.matmul(torch.softmax(sc if add is None else sc + add.to(dtype), -1), v)
        helpers.assert_no_worse_than_eager(o, ref["o"], eager, "o")
    else:
        helpers.assert_close(o, ref["o"], "o", dtype)
    helpers.assert_close(lse, ref["lse"], "lse", torch.float16, atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B", [20, 40])   # up to 32 sequences the longest come first
def test_pair_kernel_packed_batch(cuda_device, B, dtype):
    H, D, max_len, spare = 8, 128, 400, 333
    lens = [(i * 7919) % 401 for i in range(B)]
    lens[3], lens[7], lens[B - 1] = 0, 470, 128   # an empty one, one past the stated maximum, an exact tile at the end
    first = 5                                      # rows before, and `spare` rows behind, all sequences
    assert takes_pairs(B, H, max_len, max_len, packed_rows=first + sum(lens) + spare)
    cu = torch.tensor([first] + [first + sum(lens[:i + 1]) for i in range(B)], dtype=torch.int32, device=cuda_device)
    total = int(cu[-1]) + spare
    g = torch.Generator(device=cuda_device).manual_seed(5)
    q, k, v = (torch.randn(total, H, D, device=cuda_device, generator=g).to(dtype) for _ in range(3))
    o, lse = torch.ops.mha_manual.fmha_varlen_fwd(q, k, v, cu, max_len)
    covered = torch.zeros(total, dtype=torch.bool, device=cuda_device)
    for b, full in enumerate(lens):
        n, r0 = min(full, max_len), int(cu[b])
        if n == 0:
            continue
        covered[r0:r0 + n] = True
        qb, kb, vb = (x[r0:r0 + n].permute(1, 0, 2) for x in (q, k, v))
        ref = composite.attention_fp32(qb, kb, vb)
        got = o[r0:r0 + n].permute(1, 0, 2)
        if n >= 128 and dtype == torch.float16 or n >= 256:
            helpers.assert_close(got, ref["o"], f"o of {b}", dtype)
        else:
            e = torch.softmax(torch.matmul(qb, kb.transpose(-1, -2)) * D ** -0.5, -1)
            helpers.assert_no_worse_than_eager(got, ref["o"], torch.matmul(e, vb), f"o of {b}")
        helpers.assert_close(lse[:, r0:r0 + n], ref["lse"], f"lse of {b}", torch.float16, atol=1e-3, rtol=1e-4)
    assert not o[~covered].any()


@pytest.mark.parametrize("mask", ["none", "seqlen", "key"])
def test_pair_kernel_with_many_items_per_cta(cuda_device, mask):
    """Some fourteen items per CTA, pairs and single tiles by turns, so that every ring of the persistent kernel goes round; with lengths, items
    of one key step beside full ones.  Repeated calls, and calls on two streams at once, give the same bits."""
    B, H, S_q, S_k, D = 32, 16, 800, 400, 128
    assert takes_pairs(B, H, S_q, S_k)
    q, k, v = inputs(B, H, S_q, S_k, D, torch.float16, 3, cuda_device)
    lens = torch.tensor([S_k if b % 3 == 0 else 1 + 53 * b % 128 if b % 3 == 1 else 130 + 8 * b for b in range(B)], dtype=torch.int32, device=cuda_device)
    kw, add = {}, None
    if mask != "none":
        add = composite.padding_add_mask(lens, S_k)
        kw = dict(seqlens=lens) if mask == "seqlen" else dict(mask=add.reshape(B, S_k))
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    o, lse = api.fmha_forward(q, k, v, status=status, **kw)
    assert capi.check_status(status) == [0, 0, 0, 0]
    for b in range(0, B, 8):   # the reference in parts
        part = slice(b, b + 8)
        ref = composite.attention_fp32(q[part], k[part], v[part], add_mask=None if add is None else add[part])
        helpers.assert_close(o[part], ref["o"], f"o from {b}")
        helpers.assert_close(lse.view(B, H, S_q)[part], ref["lse"].view(8, H, S_q), f"lse from {b}", atol=1e-3, rtol=1e-4)
    for _ in range(10):
        again = api.fmha_forward(q, k, v, **kw)
    assert torch.equal(again[0], o) and torch.equal(again[1], lse)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    results = []
    for i in range(6):
        with torch.cuda.stream(streams[i % 2]):
            results.append(api.fmha_forward(q, k, v, **kw))
    torch.cuda.synchronize()
    assert all(torch.equal(r[0], o) and torch.equal(r[1], lse) for r in results)


@pytest.mark.parametrize("mask", ["none", "key"])
@pytest.mark.parametrize("B,H,S_q,S_k", [(1, 16, 2048, 1100), (2, 12, 1331, 1331)])   # 128 and 144 pairs, even and odd tiles per head
def test_pair_kernel_on_one_round_of_long_keys(cuda_device, B, H, S_q, S_k, mask):
    assert takes_pairs(B, H, S_q, S_k, lengths=False) and not takes_pairs(B, H, S_q, S_k)
    q, k, v = inputs(B, H, S_q, S_k, 128, torch.float16, 4, cuda_device)
    add = None if mask == "none" else torch.randn(B, S_k, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(1))
    o, lse = api.fmha_forward(q, k, v, mask=add)
    ref = composite.attention_fp32(q, k, v, add_mask=None if add is None else add.reshape(B, 1, 1, S_k))
    helpers.assert_close(o, ref["o"], "o")
    helpers.assert_close(lse, ref["lse"], "lse", atol=1e-3, rtol=1e-4)


def test_pair_kernel_on_other_layouts(cuda_device):
    """Operands and results as [B,S,H,D] views of a fused projection, results into permuted memory with room around the rows, and no
    logsumexp: the bits of the contiguous call."""
    B, H, S, D = 19, 8, 384 + 128, 128
    assert takes_pairs(B, H, S, S)
    g = torch.Generator(device=cuda_device).manual_seed(6)
    qkv = torch.randn(B, S, 3, H, D, device=cuda_device, generator=g).half()
    q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    lens = (torch.arange(B, device=cuda_device, dtype=torch.int32) * 7919) % S + 1
    o, lse = api.fmha_forward(q.contiguous(), k.contiguous(), v.contiguous(), seqlens=lens)
    o_packed, lse_packed = torch.ops.mha_manual.fmha_qkvpacked_fwd(qkv, None, lens)
    assert torch.equal(o_packed.permute(0, 2, 1, 3), o) and torch.equal(lse_packed.view_as(lse), lse)
    room = torch.full((S, B, H, 2 * D), 7.0, dtype=torch.half, device=cuda_device)
    out = room[..., :D].permute(1, 2, 0, 3)
    assert torch.equal(api.fmha_forward(q, k, v, seqlens=lens, out=out)[0], o) and (room[..., D:] == 7.0).all()
    assert torch.equal(capi.fwd(q, k, v, mask_kind=capi.MASK_SEQLEN, mask=lens, want_lse=False)["o"], o)
