"""Forward parity on the GPU: the CUDA path, called through the C ABI, against the CPU oracle
on the same seeded inputs.  Tolerance: |got - ref| <= 1e-3 + 2e-3 |ref| (see helpers.assert_close)."""
import numpy as np
import pytest
import torch

from nvfuserexamples_b200 import api, capi, sharding
from oracle import composite, philox
from tests import helpers

pytestmark = pytest.mark.gpu

SHAPES = [
    # B, H, S_q, S_k, D, dtype
    (2, 4, 128, 128, 64, torch.float16),     # the reference's own sequence length and head size
    (2, 3, 384, 384, 64, torch.float16),     # BERT-large forward shape, fewer heads
    (1, 2, 512, 512, 64, torch.bfloat16),
    (2, 2, 200, 333, 64, torch.float16),     # ragged: neither length is a tile multiple
    (1, 2, 77, 1000, 128, torch.bfloat16),
    (1, 2, 256, 384, 128, torch.float16),
    (3, 1, 1, 5, 64, torch.float16),         # a single query row, five keys
]


@pytest.mark.parametrize("B,H,S_q,S_k,D,dtype", SHAPES)
@pytest.mark.parametrize("mask", ["none", "seqlen", "key"])
def test_forward_matches_oracle(cuda_device, B, H, S_q, S_k, D, dtype, mask):
    q, k, v, _, lens = helpers.randn_like_config(B, H, S_q, S_k, D, dtype, seed=100 + S_q + S_k, device=cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    kw, okw = {}, {}
    if mask == "seqlen":
        kw["seqlens"], okw["lens"] = lens, lens
    elif mask == "key":
        add = composite.padding_add_mask(lens.cpu(), S_k).reshape(B, S_k).to(cuda_device)
        kw["mask"], okw["add_mask"] = add, add
    o, lse = api.fmha_forward(q, k, v, status=status, **kw)
    assert capi.check_status(status) == [0, 0, 0, 0]
    ref, *_ = helpers.oracle_forward(q, k, v, **okw)
    helpers.assert_close(o, ref["o"], "o", dtype)
    helpers.assert_close(lse, ref["lse"], "lse", torch.float16, atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (128, torch.bfloat16)])
@pytest.mark.parametrize("p_drop", [0.1, 0.5])
def test_forward_philox_dropout(cuda_device, D, dtype, p_drop):
    B, H, S = 2, 2, 384
    q, k, v, _, lens = helpers.randn_like_config(B, H, S, S, D, dtype, seed=7, device=cuda_device)
    o, lse = api.fmha_forward(q, k, v, seqlens=lens, p_drop=p_drop, seed=0xABCDEF12345, offset=9)
    ref, *_ = helpers.oracle_forward(q, k, v, lens=lens, p_drop=p_drop, seed=0xABCDEF12345, offset=9)
    helpers.assert_close(o, ref["o"], "o", dtype)
    helpers.assert_close(lse, ref["lse"], "lse", torch.float16, atol=1e-3, rtol=1e-4)  # lse ignores dropout


def test_dropout_mask_bit_exact(cuda_device):
    """The keep decisions taken inside the kernel, the library's device and host generators and
    the numpy restatement are the same bits."""
    B, H, S_q, S_k, p, seed, off = 1, 3, 200, 333, 0.1, 0x5EED0003, 11
    q, k, v, _, _ = helpers.randn_like_config(B, H, S_q, S_k, 64, torch.float16, seed=1, device=cuda_device)
    res = capi.fwd(q, k, v, dropout_kind=capi.DROPOUT_PHILOX, p_drop=p, seed=seed, offset=off, keep_mask_out=True)
    kernel = res["keep_mask"].cpu().numpy()
    oracle = philox.dropout_keep_mask(seed, off, 0, B * H, S_q, S_k, p)
    np.testing.assert_array_equal(kernel, oracle)
    dev = api.philox_dropout_mask(B, H, S_q, S_k, p, seed, off, device=cuda_device).cpu().numpy().reshape(B * H, S_q, S_k)
    np.testing.assert_array_equal(dev, oracle)
    np.testing.assert_array_equal(api.philox_dropout_mask(B, H, S_q, S_k, p, seed, off).reshape(B * H, S_q, S_k), oracle)
    # and the production kernel (no debug outputs) dropped the same entries as the instrumented one:
    # the two differ only by rounding, a differing keep decision would show as an O(1) difference
    o_fast, _ = api.fmha_forward(q, k, v, p_drop=p, seed=seed, offset=off)
    assert (o_fast.float() - res["o"].float()).abs().max().item() <= 2e-3


def test_tensor_memory_and_shared_memory_paths_agree(cuda_device):
    q, k, v, _, lens = helpers.randn_like_config(2, 2, 256, 384, 64, torch.float16, seed=5, device=cuda_device)
    a = capi.fwd(q, k, v, mask_kind=capi.MASK_SEQLEN, mask=lens, debug_scores=True)  # general kernel, P in tensor memory
    b = capi.fwd(q, k, v, mask_kind=capi.MASK_SEQLEN, mask=lens, flags=capi.FLAG_P_VIA_SMEM)
    assert torch.equal(a["o"], b["o"]) and torch.equal(a["lse"], b["lse"])


def test_raw_scores_are_the_fp32_gemm(cuda_device):
    q, k, v, _, _ = helpers.randn_like_config(1, 2, 128, 256, 128, torch.float16, seed=2, device=cuda_device)
    res = capi.fwd(q, k, v, debug_scores=True)
    ref = torch.matmul(q.float().cpu(), k.float().cpu().transpose(-1, -2)).reshape(2, 128, 256)
    assert (res["scores"].cpu() - ref).abs().max().item() < 1e-3


def test_edge_cases(cuda_device):
    dev = cuda_device
    torch.manual_seed(0)
    # single key: output rows equal that key's value row exactly
    q = torch.randn(1, 1, 130, 64, device=dev).half()
    k = torch.randn(1, 1, 1, 64, device=dev).half()
    v = torch.randn(1, 1, 1, 64, device=dev).half()
    o, lse = api.fmha_forward(q, k, v)
    assert torch.equal(o, v.expand(1, 1, 130, 64))
    # equal scores: mean of the values
    k8 = torch.randn(1, 1, 8, 64, device=dev).half()
    v8 = torch.randn(1, 1, 8, 64, device=dev).half()
    o, _ = api.fmha_forward(torch.zeros_like(q), k8, v8)
    helpers.assert_close(o, v8.float().mean(2, keepdim=True).expand(1, 1, 130, 64), "mean")
    # valid length 0 == nothing masked; a fully masked additive row == unmasked row (test.py:15 semantics)
    q2, k2, v2, _, _ = helpers.randn_like_config(2, 1, 64, 200, 64, torch.float16, seed=3, device=dev)
    o_none, _ = api.fmha_forward(q2, k2, v2)
    o_len0, _ = api.fmha_forward(q2, k2, v2, seqlens=torch.zeros(2, dtype=torch.int32, device=dev))
    assert torch.equal(o_none, o_len0)
    o_all, _ = api.fmha_forward(q2, k2, v2, mask=torch.full((2, 200), -10000.0, device=dev))
    helpers.assert_close(o_all, o_none.float(), "fully masked", atol=4e-3)
    # empty batch is a no-op, zero keys is an error
    api.fmha_forward(q2[:0], k2[:0], v2[:0])
    with pytest.raises(capi.FmhaError):
        api.fmha_forward(q2, k2[:, :, :0], v2[:, :, :0])


def test_strided_views_bshd(cuda_device):
    """[B,S,3,H,D] packed projections viewed as [B,H,S,D] without a copy."""
    B, S, H, D = 2, 256, 3, 64
    g = torch.Generator().manual_seed(4)
    qkv = torch.randn(B, S, 3, H, D, generator=g).half().to(cuda_device)
    q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    out = torch.empty(B, S, H, D, dtype=torch.half, device=cuda_device).permute(0, 2, 1, 3)
    o, _ = api.fmha_forward(q, k, v, out=out)
    ref, *_ = helpers.oracle_forward(q.contiguous(), k.contiguous(), v.contiguous())
    helpers.assert_close(o, ref["o"], "o strided")


def test_sharded_equals_unsharded_bitwise(cuda_device):
    B, H, S, D, p = 4, 3, 256, 64, 0.1
    q, k, v, _, lens = helpers.randn_like_config(B, H, S, S, D, torch.float16, seed=9, device=cuda_device)
    full, lse_full = api.fmha_forward(q, k, v, seqlens=lens, p_drop=p, seed=3, offset=1)
    for world in (2, 8):
        parts = []
        for r in range(world):
            sh = sharding.make_shard(B, H, world, r)
            qs, ks, vs = (sharding.shard_tensor(t, sh).contiguous() for t in (q, k, v))
            o, _ = api.fmha_forward(qs, ks, vs, seqlens=sharding.shard_per_batch(lens, sh), p_drop=p, seed=3, offset=1,
                                    bh_offset=sh.bh_offset)
            parts.append(o.reshape(sh.bh_count, S, D))
        assert torch.equal(torch.cat(parts), full.reshape(B * H, S, D))


@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (128, torch.bfloat16)])
def test_forward_is_bit_reproducible_across_calls(cuda_device, D, dtype):
    """More CTAs than resident slots, valid lengths and an additive key mask, with dropout: 40 calls give the same bits
    (nothing in the forward depends on the order in which CTAs, loads or MMAs complete)."""
    B, H, S = 8, 16, 512
    q, k, v, _, lens = helpers.randn_like_config(B, H, S, S, D, dtype, seed=12, device=cuda_device)
    add = composite.padding_add_mask(lens, S).reshape(B, S).contiguous()
    for kw in (dict(seqlens=lens), dict(mask=add)):
        first_o, first_lse = api.fmha_forward(q, k, v, p_drop=0.1, seed=4, offset=2, **kw)
        for _ in range(40):
            o, lse = api.fmha_forward(q, k, v, p_drop=0.1, seed=4, offset=2, **kw)
        assert torch.equal(o, first_o) and torch.equal(lse, first_lse)


@pytest.mark.parametrize("name", ["bert_base_fwd", "bert_large_fwd"])
def test_full_size_properties(cuda_device, name):
    """At the benchmark sizes the CPU oracle is too slow, so check size-independent properties:
    V = 1 gives O = 1 (probabilities sum to one), permuting the keys changes nothing, and one
    (batch, head) slice matches the oracle."""
    B, H, S, D, dtype, lr, p, _ = composite.CONFIGS[name]
    x = composite.make_inputs(B, H, S, D, dtype, lr, composite.CONFIG_SEEDS[name])
    q, k, v, lens = (x[n].to(cuda_device) for n in ("q", "k", "v", "lens"))
    ones = torch.ones_like(v)
    o1, lse = api.fmha_forward(q, k, ones, seqlens=lens)
    assert (o1.float() - 1).abs().max().item() <= 2e-3
    full = torch.full_like(lens, S)
    perm = torch.randperm(S, generator=torch.Generator().manual_seed(1)).to(cuda_device)
    o_a, lse_a = api.fmha_forward(q, k, v, seqlens=full)
    o_b, lse_b = api.fmha_forward(q, k[:, :, perm].contiguous(), v[:, :, perm].contiguous(), seqlens=full)
    assert (o_a.float() - o_b.float()).abs().max().item() <= 4e-3
    assert (lse_a - lse_b).abs().max().item() <= 1e-3
    b, h = B - 1, H // 2
    od, _ = api.fmha_forward(q, k, v, seqlens=lens, p_drop=p, seed=composite.PHILOX_SEEDS[name], offset=0)
    ref, *_ = helpers.oracle_forward(q[b:b + 1, h:h + 1], k[b:b + 1, h:h + 1], v[b:b + 1, h:h + 1], lens=lens[b:b + 1],
                                     p_drop=p, seed=composite.PHILOX_SEEDS[name], offset=0, bh_offset=b * H + h)
    helpers.assert_close(od[b:b + 1, h:h + 1], ref["o"], "slice o", dtype)


def test_bounded_wait_reports_instead_of_hanging(cuda_device):
    """Failure detection without faulting the GPU: a wait nothing satisfies runs out, the kernel
    returns, the status block names the site, and the context keeps working."""
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    capi.selftest_wait_timeout(status)
    with pytest.raises(capi.FmhaError) as e:
        capi.check_status(status)
    assert e.value.code == capi.FMHA_ERR_DEVICE_TIMEOUT and "900" in str(e.value)
    assert capi.check_status(status) == [0, 0, 0, 0]  # cleared by the failing check
    q, k, v, _, _ = helpers.randn_like_config(1, 1, 128, 128, 64, torch.float16, seed=1, device=cuda_device)
    o, _ = api.fmha_forward(q, k, v, status=status)
    ref, *_ = helpers.oracle_forward(q, k, v)
    helpers.assert_close(o, ref["o"], "o after timeout")


@pytest.mark.parametrize("B,H,S_q,S_k,D,dtype", [
    (1, 1, 17, 1024, 64, torch.float16),    # 8 shares of two 64-key steps
    (1, 2, 31, 1000, 64, torch.bfloat16),   # one warp of rows, a ragged last step
    (2, 2, 33, 900, 128, torch.bfloat16),   # the second warp has a single row
    (1, 1, 17, 300, 128, torch.float16),    # more shares than key steps: one of them is empty
    (1, 2, 130, 1536, 128, torch.float16),  # two query tiles, the second with two rows
    (1, 3, 128, 2048, 64, torch.float16),   # a full tile
])
@pytest.mark.parametrize("mask,p_drop", [("none", 0.0), ("seqlen", 0.1), ("key", 0.0), ("key", 0.1)])
def test_keys_split_over_a_cluster(cuda_device, B, H, S_q, S_k, D, dtype, mask, p_drop):
    """Few CTAs against long keys: the keys of a query tile are dealt out over a cluster whose CTAs combine their
    shares.  Valid lengths down to a single key leave shares without any key step.  (bf16: 130 keys, two to three steps;
    a result of one key is that key's value rounded once, up to 2^-8 of it off, which is outside assert_close's bf16 bar of
    2e-3 on 99.5 % of the elements: it presumes sums of at least 128 keys.)"""
    q, k, v, _, _ = helpers.randn_like_config(B, H, S_q, S_k, D, dtype, seed=S_q + S_k, device=cuda_device)
    lens = torch.tensor([1 if dtype == torch.float16 else 130, S_k // 2 + 3][:B], dtype=torch.int32, device=cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    kw, okw = {}, {}
    if mask == "seqlen":
        kw["seqlens"], okw["lens"] = lens, lens
    elif mask == "key":
        add = torch.randn(B, S_k, generator=torch.Generator().manual_seed(3)).to(cuda_device)
        kw["mask"], okw["add_mask"] = add, add
    o, lse = api.fmha_forward(q, k, v, p_drop=p_drop, seed=21, offset=4, status=status, **kw)
    assert capi.check_status(status) == [0, 0, 0, 0]
    ref, *_ = helpers.oracle_forward(q, k, v, p_drop=p_drop, seed=21, offset=4, **okw)
    helpers.assert_close(o, ref["o"], "o", dtype)
    helpers.assert_close(lse, ref["lse"], "lse", torch.float16, atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("B,H,S_q,S_k,D,dtype", [
    (2, 2, 1, 700, 64, torch.float16),       # one row; shares of a head over a cluster
    (1, 3, 16, 1000, 128, torch.bfloat16),   # a full 16-row tile, a ragged last step
    (2, 1, 9, 2049, 128, torch.float16),     # second half of the tile has one row; the last step has one key
    (1, 1, 15, 130, 64, torch.bfloat16),     # too few steps for shares
    (160, 1, 3, 200, 64, torch.float16),     # more heads than multiprocessors: no cluster
    (75, 16, 16, 60, 64, torch.float16),     # so many heads of so few keys that the tile kernel takes them
])
@pytest.mark.parametrize("mask,p_drop", [("none", 0.0), ("seqlen", 0.1), ("key", 0.0), ("key", 0.3)])
def test_a_handful_of_query_rows(cuda_device, B, H, S_q, S_k, D, dtype, mask, p_drop):
    """At most 16 query rows per head run on their own kernel.  (bf16: at least 130 keys, see
    test_keys_split_over_a_cluster.)  Strided operands: Q and O as [B,S,H,D], K and V as slices of one tensor."""
    g = torch.Generator().manual_seed(S_q * 7 + S_k)
    q = torch.randn(B, S_q, H, D, generator=g).to(dtype).to(cuda_device).permute(0, 2, 1, 3)
    kv = torch.randn(B, S_k, 2, H, D, generator=g).to(dtype).to(cuda_device)
    k, v = kv[:, :, 0].permute(0, 2, 1, 3), kv[:, :, 1].permute(0, 2, 1, 3)
    lens = torch.randint(1 if dtype == torch.float16 else 130, S_k + 1, (B,), generator=g, dtype=torch.int32).to(cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    kw, okw = {}, {}
    if mask == "seqlen":
        kw["seqlens"], okw["lens"] = lens, lens
    elif mask == "key":
        add = torch.randn(B, S_k, generator=g).to(cuda_device)
        kw["mask"], okw["add_mask"] = add, add
    out = torch.empty(B, S_q, H, D, dtype=dtype, device=cuda_device).permute(0, 2, 1, 3)
    o, lse = api.fmha_forward(q, k, v, p_drop=p_drop, seed=33, offset=6, bh_offset=5, status=status, out=out, **kw)
    assert capi.check_status(status) == [0, 0, 0, 0]
    ref, *_ = helpers.oracle_forward(q, k, v, p_drop=p_drop, seed=33, offset=6, bh_offset=5, **okw)
    helpers.assert_close(o, ref["o"], "o", dtype)
    helpers.assert_close(lse, ref["lse"], "lse", torch.float16, atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("p_drop", [0.0, 0.1])
def test_a_nan_among_masked_keys_is_not_stepped_over(cuda_device, D, p_drop):
    """A key whose score is NaN makes its head's rows NaN, masked away or not: NaN + mask is NaN, as in the composite.  The
    shortcut for steps whose keys are all masked away looks at the scores and must see it."""
    B, H, S = 40, 8, 512   # one CTA per query tile
    q, k, v, _, _ = helpers.randn_like_config(B, H, S, S, D, torch.float16, seed=5, device=cuda_device)
    k[3, 2, 450] = float("nan")
    mask = torch.where(torch.arange(S, device=cuda_device) < 150, 0.0, -1e4).repeat(B, 1)
    o, lse = api.fmha_forward(q, k, v, mask=mask, p_drop=p_drop, seed=1)
    assert torch.isnan(o[3, 2]).all() and torch.isnan(lse.view(B, H, S)[3, 2]).all()
    o[3, 2] = 0
    assert torch.isfinite(o).all()


@pytest.mark.parametrize("B,H,S_q,S_k", [
    (40, 8, 256, 300),    # one CTA per query tile, with a mask from tile to tile; at D = 128 two tiles per CTA
    (2, 8, 200, 300),     # one CTA per query tile at both head dimensions
    (1, 2, 130, 1536),    # keys split over a cluster
])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mask", ["none", "zero", "zero_first"])
def test_scores_of_minus_infinity_under_a_large_scale(cuda_device, B, H, S_q, S_k, D, mask):
    """Keys whose scores are all -inf contribute zeros, also where they fill a row's first step or a share of the keys and the scale is
    so large (1, as unscaled attention has it) that the lowest float times scale * log2 e is -inf itself."""
    q, k, v, _, _ = helpers.randn_like_config(B, H, S_q, S_k, D, torch.float16, seed=D + S_k, device=cuda_device)
    q, k = q * 0.35, k * 0.35   # scores of unit size, give or take, without the usual 1/sqrt(D)
    q[..., 0] = q[..., 0].abs() + 0.1
    n_inf = max(D, S_k // 8)   # at least a whole key step (64 keys at D = 64, 128 at D = 128), or a share of eight
    k[:, :, :n_inf, 0] = float("-inf")
    kw, add = {}, None
    if mask != "none":
        add = torch.zeros(B, S_k, device=cuda_device)
        if mask == "zero_first":
            add[:, n_inf:] = torch.randn(S_k - n_inf, generator=torch.Generator().manual_seed(2)).to(cuda_device)
        kw["mask"] = add
    o, lse = api.fmha_forward(q, k, v, scale=1.0, **kw)
    ref = composite.attention_fp32(q, k, v, add_mask=None if add is None else add.reshape(B, 1, 1, S_k), scale=1.0)
    helpers.assert_close(o, ref["o"], "o")
    helpers.assert_close(lse, ref["lse"], "lse", atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("B,H,S_q,S_k,D,dtype", [
    (3, 2, 200, 333, 64, torch.float16),      # one CTA per query tile
    (2, 2, 130, 520, 128, torch.bfloat16),
    (1, 2, 130, 1536, 128, torch.float16),    # keys split over a cluster: whole shares before the first live key
    (19, 8, 256, 520, 128, torch.float16),    # two query tiles per CTA
])
@pytest.mark.parametrize("pad", [-10000.0, float("-inf")])
@pytest.mark.parametrize("p_drop", [0.0, 0.1])
def test_additive_mask_that_pads_on_the_left(cuda_device, B, H, S_q, S_k, D, dtype, pad, p_drop):
    """Whole key steps are masked away before the first live key, and, in the second batch element, between live keys."""
    if B > 4 and p_drop > 0:
        B, H = 2, 2   # with dropout the kernel of one tile takes any grid, and the oracle draws on the CPU
    q, k, v, _, _ = helpers.randn_like_config(B, H, S_q, S_k, D, dtype, seed=S_k, device=cuda_device)
    add = torch.zeros(B, S_k)
    for b in range(B):
        add[b, :S_k - 130 - 7 * b] = pad
    if B > 1:
        add[1, :3] = 0.5
    add = add.to(cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    o, lse = api.fmha_forward(q, k, v, mask=add, p_drop=p_drop, seed=8, offset=3, status=status)
    assert capi.check_status(status) == [0, 0, 0, 0]
    ref, *_ = helpers.oracle_forward(q, k, v, add_mask=add, p_drop=p_drop, seed=8, offset=3)
    helpers.assert_close(o, ref["o"], "o", dtype)
    helpers.assert_close(lse, ref["lse"], "lse", torch.float16, atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("p", [0.0, 0.2])
@pytest.mark.parametrize("mask", ["none", "seqlen", "key"])
@pytest.mark.parametrize("S_k,D", [(31, 64), (32, 64), (33, 64), (63, 64), (65, 64), (95, 64), (96, 64), (97, 64),
                                   (63, 128), (64, 128), (65, 128), (127, 128), (129, 128), (191, 128), (192, 128), (193, 128)])
def test_last_key_step_around_half_a_step(cuda_device, S_k, D, mask, p):
    """A last step of up to 32 keys (64 at head dimension 128) is done by halves; lengths around it, and whole steps past a length."""
    B, H, S_q, dtype = 4, 2, 130, torch.float16
    q, k, v, _, _ = helpers.randn_like_config(B, H, S_q, S_k, D, dtype, seed=S_k, device=cuda_device)
    lens = torch.tensor([S_k, max(1, S_k - 1), max(1, S_k - D // 2 + 1), max(1, S_k - D // 2 - 1)], dtype=torch.int32, device=cuda_device)
    kw, okw = {}, {}
    if mask == "seqlen":
        kw["seqlens"], okw["lens"] = lens, lens
    elif mask == "key":
        add = composite.padding_add_mask(lens.cpu(), S_k).reshape(B, S_k).to(cuda_device)
        kw["mask"], okw["add_mask"] = add, add
    o, lse = api.fmha_forward(q, k, v, p_drop=p, seed=4, offset=9, **kw)
    ref, *_ = helpers.oracle_forward(q, k, v, p_drop=p, seed=4, offset=9, **okw)
    helpers.assert_close(o, ref["o"], "o", dtype)
    helpers.assert_close(lse, ref["lse"], "lse", torch.float16, atol=1e-3, rtol=1e-4)
