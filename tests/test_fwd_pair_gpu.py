"""The forward kernel for grids that fill the chip (two query tiles per CTA, persistent) against the fp32 composite: even and
odd numbers of query tiles, key counts around the key step, every mask kind, and packed batches with empty
sequences, sequences past the stated maximum and rows outside all sequences.  Tolerances: helpers.assert_close."""
import pytest
import torch

import mha_manual  # noqa: F401  registers torch.ops.mha_manual.*
from nvfuserexamples_b200 import api, capi
from oracle import composite
from tests import helpers

pytestmark = pytest.mark.gpu


def inputs(B, H, S_q, S_k, D, dtype, seed, dev):
    g = torch.Generator(device=dev).manual_seed(seed)
    r = lambda S: torch.randn(B, H, S, D, device=dev, generator=g).to(dtype)
    return r(S_q), r(S_k), r(S_k)


def takes_pairs(heads, S_q, S_k):   # the library's rule (fwd_pair_applies), so that the sizes below keep to it
    sms, n = torch.cuda.get_device_properties(0).multi_processor_count, (S_q + 127) // 128
    pair_rounds, tile_rounds = -(-heads * ((n + 1) // 2) // sms), -(-heads * n // (2 * sms))
    return S_k > 256 and heads * n >= 2 * sms and 7 * pair_rounds <= 8 * tile_rounds


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("mask", ["none", "seqlen", "key", "key_inf"])
@pytest.mark.parametrize("B,H,S_q,S_k", [(37, 4, 129, 257), (19, 8, 256, 384), (13, 8, 300, 385), (8, 8, 640, 511), (19, 8, 200, 900)])
def test_pair_kernel_matches_the_composite(cuda_device, B, H, S_q, S_k, mask, dtype):
    D = 128
    assert takes_pairs(B * H, S_q, S_k)
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
    assert takes_pairs(B * H, max_len, max_len)
    first = 5                                      # rows before, and `spare` rows behind, all sequences
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
