"""The forward kernel whose CTAs go from query tile to query tile (head dimension 64, large grids) against the kernel of one tile per
CTA, bit for bit, on the same batch in pieces too small for it, and against the fp32 composite: one key step and several, last
steps of up to and more than half a step, ragged query tiles, each mask kind, dropout.  Tolerances: helpers.assert_close."""
import pytest
import torch

import mha_manual  # noqa: F401  registers torch.ops.mha_manual.*
from nvfuserexamples_b200 import api, capi
from oracle import composite
from tests import helpers
from tests.test_fwd_rules import chain_pays

pytestmark = pytest.mark.gpu

B, H, PIECE = 75, 12, 15   # two query tiles per head: 1 800 tiles; 360 in a piece, where the keys of a tile are not split over a cluster either


def batch(S_q, S_k, dtype, kind, dev):
    g = torch.Generator(device=dev).manual_seed(S_q + S_k)
    q, k, v = (torch.randn(B, H, S, 64, device=dev, generator=g).to(dtype) for S in (S_q, S_k, S_k))
    lens = (torch.arange(B, device=dev, dtype=torch.int32) * 7919) % S_k + 1
    if kind == "seqlen":
        return q, k, v, dict(seqlens=lens), composite.padding_add_mask(lens, S_k)
    if kind == "key":   # padding at the end, at the start, -inf, and none
        add = composite.padding_add_mask(lens, S_k, -10000.0).reshape(B, S_k)
        add[1::4] = add[1::4].flip(-1)
        add[2::4] = torch.where(add[2::4] < 0, float("-inf"), 0.0)
        add[3::4] = 0.0
        return q, k, v, dict(mask=add), add.reshape(B, 1, 1, S_k)
    return q, k, v, {}, None


@pytest.mark.parametrize("p", [0.0, 0.2])
@pytest.mark.parametrize("kind", ["none", "seqlen", "key"])
@pytest.mark.parametrize("S_q,S_k", [(129, 1), (200, 32), (129, 33), (256, 64), (129, 65), (140, 97), (129, 160), (255, 250)])
def test_same_bits_as_a_tile_per_cta(cuda_device, S_q, S_k, kind, p):
    dtype = torch.float16 if (S_q + S_k) % 2 else torch.bfloat16
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert chain_pays(sms, B * H * 2, S_k, kind == "key", p > 0) and not chain_pays(sms, PIECE * H * 2, S_k, kind == "key", p > 0)
    q, k, v, kw, add = batch(S_q, S_k, dtype, kind, cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    o, lse = api.fmha_forward(q, k, v, p_drop=p, seed=5, offset=2, status=status, **kw)
    assert capi.check_status(status) == [0, 0, 0, 0]
    for b in range(0, B, PIECE):
        s = slice(b, b + PIECE)
        op, lp = api.fmha_forward(q[s], k[s], v[s], p_drop=p, seed=5, offset=2, bh_offset=b * H, **{n: t[s] for n, t in kw.items()})
        assert torch.equal(o[s], op) and torch.equal(lse[s], lp)
    if p == 0.0 and dtype == torch.float16:
        ref = composite.attention_fp32(q, k, v, add_mask=add)
        helpers.assert_close(o, ref["o"], "o", dtype)
        helpers.assert_close(lse, ref["lse"], "lse", torch.float16, atol=1e-3, rtol=1e-4)


def test_repeated_and_concurrent_calls(cuda_device):
    """Calls on two streams share the SMs, so that a call's CTAs start at any time; every result is the same."""
    q, k, v, kw, _ = batch(256, 128, torch.float16, "seqlen", cuda_device)
    first = api.fmha_forward(q, k, v, p_drop=0.1, seed=1, offset=1, **kw)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for i in range(6):
        with torch.cuda.stream(streams[i % 2]):
            got.append(api.fmha_forward(q, k, v, p_drop=0.1, seed=1, offset=1, **kw))
    torch.cuda.synchronize()
    for o, lse in got:
        assert torch.equal(o, first[0]) and torch.equal(lse, first[1])


@pytest.mark.parametrize("kind,p", [("none", 0.0), ("seqlen", 0.2), ("key", 0.0)])
def test_fused_projection_layout_and_strided_out(cuda_device, kind, p):
    """q, k and v as views of one [B,S,3,H,D] tensor, O into a view of a larger buffer: the bits of the call on contiguous tensors, and nothing beside them."""
    S = 140
    q, k, v, kw, _ = batch(S, S, torch.bfloat16, kind, cuda_device)
    want = api.fmha_forward(q, k, v, p_drop=p, seed=5, offset=2, **kw)
    qkv = torch.stack([t.transpose(1, 2) for t in (q, k, v)], dim=2)
    buf = torch.full((B, S + 9, H + 1, 64), 7.0, dtype=torch.bfloat16, device=cuda_device)
    o, lse = api.fmha_forward(*(qkv[:, :, i].transpose(1, 2) for i in range(3)), p_drop=p, seed=5, offset=2, out=buf[:, :S, :H].transpose(1, 2), **kw)
    assert torch.equal(o, want[0]) and torch.equal(lse, want[1])
    assert (buf[:, S:] == 7.0).all() and (buf[:, :, H] == 7.0).all()


def test_replayed_graph_and_device_resident_offset(cuda_device):
    """A captured call replays with the bits of an eager one, the Philox offset from the value the tensor holds then."""
    ops = torch.ops.mha_manual
    q, k, v, kw, _ = batch(256, 128, torch.float16, "seqlen", cuda_device)
    lens, off = kw["seqlens"], torch.zeros(1, dtype=torch.int64, device=cuda_device)
    eager = {value: ops.fmha_fwd(q, k, v, None, lens, 0.2, 3, 10 + value) for value in (0, 5)}
    torch.cuda.synchronize()
    side = torch.cuda.Stream(device=cuda_device)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            o, lse = ops.fmha_fwd(q, k, v, None, lens, 0.2, 3, 10, None, 0, off)
    torch.cuda.current_stream().wait_stream(side)
    for value in (0, 5, 0):
        off.fill_(value)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(o, eager[value][0]) and torch.equal(lse, eager[value][1])
    assert not torch.equal(eager[0][0], eager[5][0])
    ops.check_status()


@pytest.mark.parametrize("p", [0.0, 0.2])
def test_a_nan_among_masked_keys_is_not_stepped_over(cuda_device, p):
    """As in the kernel of one tile per CTA: a key whose score is NaN makes its head's rows NaN, masked away or not, and no other head's."""
    S = 250
    q, k, v, _, _ = batch(S, S, torch.float16, "none", cuda_device)
    mask = torch.where(torch.arange(S, device=cuda_device) < 50, 0.0, -1e4).repeat(B, 1)
    want, _ = api.fmha_forward(q, k, v, mask=mask, p_drop=p, seed=1)
    k[30, 5, 200] = float("nan")
    o, lse = api.fmha_forward(q, k, v, mask=mask, p_drop=p, seed=1)
    assert torch.isnan(o[30, 5]).all() and torch.isnan(lse.view(B, H, S)[30, 5]).all()
    o[30, 5] = want[30, 5]
    assert torch.isfinite(want).all() and torch.equal(o, want)
