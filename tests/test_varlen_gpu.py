"""Packed variable-length batches (FMHA_MASK_CU_SEQLENS) against the fp32 oracle, sequence by sequence.

The reference lists padded / irregular shapes as open work (fmha/fmha_manual.cpp:110, :178 of
shmsong/NvFuserExamples); here a batch is one [total_rows, H, D] tensor per operand plus row offsets."""
import ctypes as C

import pytest
import torch

from nvfuserexamples_b200 import capi
from tests import helpers

pytestmark = pytest.mark.gpu


def packed_batch(lens, H, D, dtype, seed, device):
    g = torch.Generator().manual_seed(seed)
    total = sum(lens)
    q, k, v, d_o = (torch.randn(total, H, D, generator=g).to(dtype).to(device) for _ in range(4))
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=device)
    return q, k, v, d_o, cu


def per_sequence_oracle(q, k, v, d_o, lens, p_drop, seed, offset, max_len):
    """Runs the composite (and its autograd backward) on every sequence alone.  The dropout mask of
    sequence b is rows/columns [0, len_b) of the mask the padded batch would draw."""
    H = q.shape[1]
    outs = {n: [] for n in ("o", "lse", "dq", "dk", "dv")}
    keep_all = helpers.keep_mask(seed, offset, 0, len(lens), H, max_len, max_len, p_drop) if p_drop > 0 else None
    ks = helpers.philox.keep_scale(p_drop) if p_drop > 0 else 1.0
    r0 = 0
    for b, n in enumerate(lens):
        if n == 0:
            continue
        sl = slice(r0, r0 + n)
        qb, kb, vb, dob = (x[sl].permute(1, 0, 2).unsqueeze(0).cpu() for x in (q, k, v, d_o))   # [1,H,n,D]
        keep = keep_all[b:b + 1, :, :n, :n] if keep_all is not None else None
        ref = helpers.composite.attention_fp32(qb, kb, vb, add_mask=None, keep=keep, keep_scale=ks)
        dq, dk, dv = helpers.composite.attention_grads_fp32(qb, kb, vb, dob, add_mask=None, keep=keep, keep_scale=ks)
        outs["o"].append(ref["o"][0].permute(1, 0, 2))
        outs["lse"].append(ref["lse"][0])                     # [H, n]
        for name, t in (("dq", dq), ("dk", dk), ("dv", dv)):
            outs[name].append(t[0].permute(1, 0, 2))
        r0 += n
    return {"o": torch.cat(outs["o"]), "lse": torch.cat(outs["lse"], dim=1), "dq": torch.cat(outs["dq"]),
            "dk": torch.cat(outs["dk"]), "dv": torch.cat(outs["dv"])}


@pytest.mark.parametrize("D,dtype,p_drop", [(64, torch.float16, 0.0), (64, torch.float16, 0.1),
                                            (128, torch.bfloat16, 0.0), (128, torch.float16, 0.1)])
def test_packed_batch_matches_the_oracle_per_sequence(cuda_device, D, dtype, p_drop):
    lens = [200, 77, 128, 1, 333, 256]      # partial tiles, an exact tile, a single row, multiples of the tile
    H, max_len = 3, 384
    q, k, v, d_o, cu = packed_batch(lens, H, D, dtype, seed=21, device=cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    canary = 7.0
    o = torch.full_like(q, canary)
    res = capi.fwd_varlen(q, k, v, cu, max_len, p_drop=p_drop, seed=5, offset=2, status=status, out=o)
    dq, dk, dv = capi.bwd_varlen(d_o, q, k, v, res["o"], res["lse"], cu, max_len, p_drop=p_drop, seed=5, offset=2,
                                 status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    ref = per_sequence_oracle(q, k, v, d_o, lens, p_drop, 5, 2, max_len)
    helpers.assert_close(res["o"], ref["o"], "o", dtype)
    helpers.assert_close(res["lse"], ref["lse"], "lse", torch.float16, atol=2e-3)
    helpers.assert_close(dq, ref["dq"], "dq", dtype)
    helpers.assert_close(dk, ref["dk"], "dk", dtype)
    helpers.assert_close(dv, ref["dv"], "dv", dtype)


@pytest.mark.parametrize("i", range(10))
def test_packed_batches_of_random_composition(cuda_device, i):
    """Seeded random numbers of sequences, lengths (empty ones included), heads, head dimension and dropout."""
    g = torch.Generator().manual_seed(2000 + i)
    r = lambda lo, hi: int(torch.randint(lo, hi + 1, (1,), generator=g))
    lens = [r(0, 400) if r(0, 5) else 0 for _ in range(r(1, 7))]
    if sum(lens) == 0:
        lens[0] = 37
    H, D, p_drop = r(1, 4), (64, 128)[r(0, 1)], (0.0, 0.1, 0.3)[r(0, 2)]
    max_len = max(lens)
    q, k, v, d_o, cu = packed_batch(lens, H, D, torch.float16, seed=300 + i, device=cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    res = capi.fwd_varlen(q, k, v, cu, max_len, p_drop=p_drop, seed=9, offset=i, status=status)
    dq, dk, dv = capi.bwd_varlen(d_o, q, k, v, res["o"], res["lse"], cu, max_len, p_drop=p_drop, seed=9, offset=i,
                                 status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    ref = per_sequence_oracle(q, k, v, d_o, lens, p_drop, 9, i, max_len)
    for name, got in (("o", res["o"]), ("dq", dq), ("dk", dk), ("dv", dv)):
        # a sequence of one row: dS cancels exactly and dQ is the rounding of delta (see the single-key note of the backward tests)
        helpers.assert_close(got, ref[name], f"{name} lens={lens}", atol=4e-3 if (name == "dq" and 1 in lens and p_drop > 0) else helpers.ATOL)


def test_packed_batch_with_more_work_items_than_sms(cuda_device):
    """48 sequences x 8 heads x up to 3 key tiles: every persistent CTA handles several items of different
    lengths; two sequences are checked against the oracle on their own."""
    g = torch.Generator().manual_seed(17)
    lens = torch.randint(1, 385, (48,), generator=g).tolist()
    H, D = 8, 64
    q, k, v, d_o, cu = packed_batch(lens, H, D, torch.float16, seed=23, device=cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    res = capi.fwd_varlen(q, k, v, cu, 384, status=status)
    dq, dk, dv = capi.bwd_varlen(d_o, q, k, v, res["o"], res["lse"], cu, 384, status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    for b in (0, 29, 47):
        sl = slice(starts[b], starts[b + 1])
        ref = per_sequence_oracle(q[sl], k[sl], v[sl], d_o[sl], [lens[b]], 0.0, 0, 0, 384)
        helpers.assert_close(res["o"][sl], ref["o"], f"o[{b}]")
        helpers.assert_close(dq[sl], ref["dq"], f"dq[{b}]")
        helpers.assert_close(dk[sl], ref["dk"], f"dk[{b}]")
        helpers.assert_close(dv[sl], ref["dv"], f"dv[{b}]")


def test_packed_batch_equals_the_padded_batch_on_its_valid_rows(cuda_device):
    """Forward outputs of the packed call are bit-identical to the padded call with valid lengths:
    same tiles, same arithmetic, same Philox bits."""
    lens = [130, 64, 255]
    H, D, S = 2, 64, 256
    q, k, v, _, cu = packed_batch(lens, H, D, torch.float16, seed=3, device=cuda_device)
    res = capi.fwd_varlen(q, k, v, cu, S, p_drop=0.1, seed=9, offset=1)
    qp, kp, vp = (torch.zeros(len(lens), H, S, D, dtype=torch.float16, device=cuda_device) for _ in range(3))
    r0 = 0
    for b, n in enumerate(lens):
        for dst, src in ((qp, q), (kp, k), (vp, v)):
            dst[b, :, :n] = src[r0:r0 + n].permute(1, 0, 2)
        r0 += n
    lens_t = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    pad = capi.fwd(qp, kp, vp, mask_kind=capi.MASK_SEQLEN, mask=lens_t, dropout_kind=capi.DROPOUT_PHILOX, p_drop=0.1,
                   seed=9, offset=1)
    r0 = 0
    for b, n in enumerate(lens):
        assert torch.equal(res["o"][r0:r0 + n].permute(1, 0, 2), pad["o"][b, :, :n])
        assert torch.equal(res["lse"][:, r0:r0 + n], pad["lse"][b, :, :n])
        r0 += n


def test_packed_batch_with_empty_sequences(cuda_device):
    """Sequences of length zero own no rows and produce nothing; their neighbours are unaffected."""
    lens = [0, 130, 0, 0, 40, 0]
    H, D = 2, 64
    q, k, v, d_o, cu = packed_batch(lens, H, D, torch.float16, seed=8, device=cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    res = capi.fwd_varlen(q, k, v, cu, 256, p_drop=0.1, seed=2, offset=1, status=status)
    dq, dk, dv = capi.bwd_varlen(d_o, q, k, v, res["o"], res["lse"], cu, 256, p_drop=0.1, seed=2, offset=1, status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    ref = per_sequence_oracle(q, k, v, d_o, lens, 0.1, 2, 1, 256)
    helpers.assert_close(res["o"], ref["o"], "o")
    helpers.assert_close(dq, ref["dq"], "dq")
    helpers.assert_close(dk, ref["dk"], "dk")
    helpers.assert_close(dv, ref["dv"], "dv")


def test_packed_batch_leaves_neighbouring_rows_alone(cuda_device):
    """A sequence's last, partial tile must not write into the next sequence (or past the end)."""
    lens = [5, 300, 60]
    H, D = 2, 64
    q, k, v, d_o, cu = packed_batch(lens, H, D, torch.float16, seed=4, device=cuda_device)
    total = sum(lens)
    # outputs with guard rows behind the packed rows
    o = torch.full((total + 64, H, D), 3.0, dtype=torch.float16, device=cuda_device)
    res = capi.fwd_varlen(q, k, v, cu, 384, out=o[:total])
    torch.cuda.synchronize()
    assert (o[total:] == 3.0).all()
    ref = per_sequence_oracle(q, k, v, d_o, lens, 0.0, 0, 0, 384)
    helpers.assert_close(res["o"], ref["o"], "o")


def test_packed_autograd_operator(cuda_device):
    import mha_manual  # noqa: F401
    ops = torch.ops.mha_manual
    lens = [150, 40, 257]
    H, D = 2, 64
    q, k, v, d_o, cu = packed_batch(lens, H, D, torch.float16, seed=12, device=cuda_device)
    q.requires_grad_(True); k.requires_grad_(True); v.requires_grad_(True)
    o = ops.fmha_varlen(q, k, v, cu, 384, 0.1, 77, 4)
    o.backward(d_o)
    ref = per_sequence_oracle(q.detach(), k.detach(), v.detach(), d_o, lens, 0.1, 77, 4, 384)
    helpers.assert_close(o, ref["o"], "o")
    helpers.assert_close(q.grad, ref["dq"], "dq")
    helpers.assert_close(k.grad, ref["dk"], "dk")
    helpers.assert_close(v.grad, ref["dv"], "dv")
    # the device-resident offset is added to the launch parameter: 1 + 3 draws the bits of offset 4
    off = torch.full((1,), 3, dtype=torch.int64, device=cuda_device)
    o2, _ = ops.fmha_varlen_fwd(q.detach(), k.detach(), v.detach(), cu, 384, 0.1, 77, 1, None, off)
    assert torch.equal(o2, o.detach())
    ops.check_status()


def test_packed_batch_on_the_fused_projection_layout(cuda_device):
    """qkv [total_rows,3,H,D] in, o [total_rows,H,D] out, one [total_rows,3,H,D] gradient back; sequences that
    end inside a tile exercise the row-wise edge stores through the strided layout."""
    import mha_manual  # noqa: F401
    ops = torch.ops.mha_manual
    lens = [150, 0, 40, 257, 128]
    H, D, p = 3, 64, 0.1
    q, k, v, d_o, cu = packed_batch(lens, H, D, torch.float16, seed=31, device=cuda_device)
    qkv = torch.stack((q, k, v), dim=1).contiguous().requires_grad_()     # [total, 3, H, D]
    o = ops.fmha_varlen_qkvpacked(qkv, cu, 384, p, 77, 4)
    assert o.shape == q.shape and o.is_contiguous()
    (dqkv,) = torch.autograd.grad(o, (qkv,), d_o)
    assert dqkv.shape == qkv.shape and dqkv.is_contiguous()
    ops.check_status()
    ref = per_sequence_oracle(q, k, v, d_o, lens, p, 77, 4, 384)
    helpers.assert_close(o, ref["o"], "o")
    for i, name in enumerate(("dq", "dk", "dv")):
        helpers.assert_close(dqkv[:, i], ref[name], name)
    # the same bits as the three-tensor operator
    o2, _ = ops.fmha_varlen_fwd(q, k, v, cu, 384, p, 77, 4)
    assert torch.equal(o2, o.detach())


def test_sequence_longer_than_max_seqlen_is_cut_not_spilled(cuda_device):
    """A sequence longer than the stated max_seqlen is processed up to max_seqlen (queries and keys alike) and its
    rows past that are left alone; above all, nothing of it lands in its neighbours' outputs or gradients (the dQ
    accumulator and delta rows of the next head lie right behind max_seqlen)."""
    import mha_manual  # noqa: F401
    lens, max_len, H, D, dtype = [150, 300, 90], 256, 2, 64, torch.float16
    q, k, v, d_o, cu = packed_batch(lens, H, D, dtype, seed=33, device=cuda_device)
    # what it must equal: the same batch with the long sequence cut to its first max_seqlen rows
    keep_rows = torch.cat([torch.arange(0, 150), torch.arange(150, 150 + 256), torch.arange(450, 540)]).to(cuda_device)
    cut = [150, 256, 90]
    qc, kc, vc, doc = (x[keep_rows].contiguous() for x in (q, k, v, d_o))
    ref = per_sequence_oracle(qc, kc, vc, doc, cut, 0.0, 0, 0, max_len)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    canary = 7.0
    o = torch.full_like(q, canary)
    res = capi.fwd_varlen(q, k, v, cu, max_len, status=status, out=o)
    dq, dk, dv = capi.bwd_varlen(d_o, q, k, v, res["o"], res["lse"], cu, max_len, status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0]
    helpers.assert_close(res["o"][keep_rows], ref["o"], "o", dtype)
    assert (res["o"][406:450] == canary).all(), "rows past max_seqlen were written"
    helpers.assert_close(dq[keep_rows], ref["dq"], "dq", dtype)
    helpers.assert_close(dk[keep_rows], ref["dk"], "dk", dtype)
    helpers.assert_close(dv[keep_rows], ref["dv"], "dv", dtype)
    # the torch operators hand back zeros for the rows that are not computed
    ops = torch.ops.mha_manual
    o2, lse2 = ops.fmha_varlen_fwd(q, k, v, cu, max_len)
    g = ops.fmha_varlen_bwd(d_o, q, k, v, o2, lse2, cu, max_len)
    assert (o2[406:450] == 0).all() and all((t[406:450] == 0).all() for t in g)
    helpers.assert_close(g[0][keep_rows], ref["dq"], "dq (operator)", dtype)


@pytest.mark.parametrize("lens,gap,tail,max_len", [([150, 300, 90], 0, 0, 256), ([40, 130], 7, 33, 128), ([128], 1, 0, 128), ([0, 5], 0, 9, 64),
                                                   ([40, 130], 700, 3001, 128), ([5], 0, 20000, 64), ([1500, 0, 20], 1, 400, 100),
                                                   ([300, 10, 0, 64, 200], 5, 100, 256), ([100] * 9, 3, 30, 104)])
@pytest.mark.parametrize("D", [64, 128])
def test_operators_zero_the_rows_no_tile_covers(cuda_device, lens, gap, tail, max_len, D):
    """Rows past max_seqlen of their sequence and rows outside all sequences are zeros whatever the memory held before
    (blocks of NaN are handed back to the caching allocator first); every other row is finite."""
    import mha_manual  # noqa: F401
    H, total = 3, gap + sum(lens) + tail
    q, k, v, d_o = (torch.randn(total, H, D, device=cuda_device).half() for _ in range(4))
    cu = [gap]
    for n in lens:
        cu.append(cu[-1] + n)
    covered = torch.zeros(total, dtype=torch.bool)
    for i, n in enumerate(lens):
        covered[cu[i]:cu[i] + min(n, max_len)] = True
    cu = torch.tensor(cu, dtype=torch.int32, device=cuda_device)
    ops = torch.ops.mha_manual

    def poison():
        x = [torch.full_like(q, float("nan")) for _ in range(8)]
        del x

    poison()
    o, lse = ops.fmha_varlen_fwd(q, k, v, cu, max_len)
    poison()
    for t in (o, *ops.fmha_varlen_bwd(d_o, q, k, v, o, lse, cu, max_len)):
        t = t.cpu()
        assert (t[~covered] == 0).all() and torch.isfinite(t[covered]).all()


@pytest.mark.parametrize("B,H,S", [(2, 25, 260), (31, 5, 65), (32, 3, 300), (32, 37, 128)])
def test_sequences_taken_longest_first_give_the_same_bits(cuda_device, B, H, S):
    """Up to 32 sequences in more CTAs than SMs are taken longest first, whatever their order in the batch; the same batch
    with sequences added up to 33 is not.  Each CTA's arithmetic is the same: the same bits.  Lengths 0 (nothing masked),
    past the end, 1, equal ones; packed: also an empty sequence."""
    dtype = torch.float16
    g = torch.Generator().manual_seed(B)
    lens = torch.randint(1, S + 1, (33,), generator=g, dtype=torch.int32)
    lens[:2] = torch.tensor([1, S])
    if B > 8:
        lens[2:8] = torch.tensor([0, S + 40, S // 2, S // 2, S // 2 + 1, S])
    q, k, v = (torch.randn(33, H, S, 64, generator=g).to(dtype).to(cuda_device) for _ in range(3))
    dev = lens.to(cuda_device)
    few = capi.fwd(q[:B], k[:B], v[:B], mask_kind=capi.MASK_SEQLEN, mask=dev[:B].contiguous())
    all33 = capi.fwd(q, k, v, mask_kind=capi.MASK_SEQLEN, mask=dev)
    assert torch.equal(few["o"], all33["o"][:B]) and torch.equal(few["lse"].view(-1), all33["lse"].view(-1)[:B * H * S])
    ops = torch.ops.mha_manual
    n = [min(int(x), S) for x in lens]
    cu = torch.tensor([0] + list(torch.tensor(n).cumsum(0)), dtype=torch.int32, device=cuda_device)
    pq, pk, pv = (torch.cat([t[b, :, :n[b]].transpose(0, 1) for b in range(33)]).contiguous() for t in (q, k, v))
    rows = int(cu[B])
    o1, lse1 = ops.fmha_varlen_fwd(pq[:rows].contiguous(), pk[:rows].contiguous(), pv[:rows].contiguous(), cu[:B + 1].contiguous(), S)
    o2, lse2 = ops.fmha_varlen_fwd(pq, pk, pv, cu, S)
    assert torch.equal(o1, o2[:rows]) and torch.equal(lse1, lse2[:, :rows])
    for b in (0, 1, B - 1):
        if n[b] >= 128:   # sums long enough for the oracle's bar
            ref, *_ = helpers.oracle_forward(q[b:b + 1], k[b:b + 1], v[b:b + 1], lens=lens[b:b + 1].clamp(max=S))
            helpers.assert_close(few["o"][b:b + 1], ref["o"], f"o[{b}]", dtype)


def test_deterministic_algorithms_fill_what_no_sequence_writes(cuda_device):
    """torch.use_deterministic_algorithms fills new memory with NaN: the logsumexp rows outside all sequences."""
    import mha_manual  # noqa: F401
    x = torch.randn(3, 200, 2, 64, device=cuda_device).half()
    cu = torch.tensor([10, 150], dtype=torch.int32, device=cuda_device)
    lse = torch.zeros(2, 200, device=cuda_device)   # the block the operator's allocation is likely to get
    del lse
    before = torch.are_deterministic_algorithms_enabled(), torch.utils.deterministic.fill_uninitialized_memory
    try:
        torch.use_deterministic_algorithms(True, warn_only=True)
        torch.utils.deterministic.fill_uninitialized_memory = True
        lse = torch.ops.mha_manual.fmha_varlen_fwd(x[0], x[1], x[2], cu, 200)[1].cpu()
    finally:
        torch.use_deterministic_algorithms(before[0])
        torch.utils.deterministic.fill_uninitialized_memory = before[1]
    assert torch.isnan(lse[:, :10]).all() and torch.isnan(lse[:, 150:]).all() and torch.isfinite(lse[:, 10:150]).all()


@pytest.mark.parametrize("D", [64, 128])
def test_uncovered_rows_are_zeroed_inside_the_tensor_only(cuda_device, D):
    """Offsets that reach past the rows the call states (a caller's mistake the host cannot see): the zeroing of uncovered
    rows stops at the last of them.  The tensors are the first 200 rows of larger ones."""
    H, total, room, max_len = 2, 200, 320, 64
    q, k, v, d_o = (torch.randn(room, H, D, device=cuda_device).half() for _ in range(4))
    cu = torch.tensor([0, 100, 300], dtype=torch.int32, device=cuda_device)   # covered: 0..63 and 100..163
    outs = [torch.full((room, H, D), 7.0, dtype=torch.float16, device=cuda_device) for _ in range(4)]
    r = capi.fwd_varlen(q[:total], k[:total], v[:total], cu, max_len, out=outs[0][:total], flags=capi.FLAG_ZERO_UNCOVERED)
    capi.bwd_varlen(d_o[:total], q[:total], k[:total], v[:total], r["o"], r["lse"], cu, max_len,
                    out=tuple(t[:total] for t in outs[1:]), flags=capi.FLAG_ZERO_UNCOVERED)
    for t in outs:
        assert (t[total:] == 7.0).all() and (t[164:total] == 0).all() and (t[64:100] == 0).all() and torch.isfinite(t).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H", [(3, 2), (60, 8)])   # one CTA per query tile; at D = 128 two
def test_forward_writes_inside_the_tensor_only(cuda_device, B, H, D):
    """Offsets that reach past the tensor, which the host cannot see: neither O nor logsumexp is written behind its end.  (The tensors are the
    first rows of larger buffers.)  The rows of the other sequences, and those of the one that is cut, are as they should be."""
    max_len, spare = 400, 900
    lens = [300] * (B - 2) + [400, 400]
    cu_list = [0]
    for n in lens:
        cu_list.append(cu_list[-1] + n)
    total = cu_list[-2] - 260   # the last but one ends 260 rows past the tensor, the last one begins there
    cu = torch.tensor(cu_list, dtype=torch.int32, device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(7)
    q, k, v = (torch.randn(total, H, D, device=cuda_device, generator=g).half() for _ in range(3))
    o = torch.full((total + spare, H, D), 7.0, dtype=torch.half, device=cuda_device)
    lse = torch.full((H * total + spare,), 7.0, device=cuda_device)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    p = capi.FwdParams()
    p.struct_bytes, p.dtype = C.sizeof(capi.FwdParams), capi.DTYPE_F16
    p.B, p.H, p.S_q, p.S_k, p.D, p.scale, p.total_rows = B, H, max_len, max_len, D, D ** -0.5, total
    p.q, p.k, p.v, p.o = (capi.Tensor4(t.data_ptr(), 0, D, H * D) for t in (q, k, v, o))
    p.lse, p.mask_kind, p.mask, p.status = lse.data_ptr(), capi.MASK_CU_SEQLENS, cu.data_ptr(), status.data_ptr()
    assert capi.load().fmha_sm100_fwd(C.byref(p), torch.cuda.current_stream().cuda_stream) == capi.FMHA_OK
    assert capi.check_status(status) == [0, 0, 0, 0]
    assert (o[total:] == 7.0).all() and (lse[H * total:] == 7.0).all()
    for b in (0, B - 3, B - 2):
        r0, rows = cu_list[b], min(lens[b], total - cu_list[b])
        qb, kb, vb = (torch.nn.functional.pad(x[r0:r0 + rows], (0, 0, 0, 0, 0, lens[b] - rows)).permute(1, 0, 2) for x in (q, k, v))
        ref = helpers.composite.attention_fp32(qb, kb, vb)
        helpers.assert_close(o[r0:r0 + rows].permute(1, 0, 2), ref["o"][:, :rows], f"o of {b}")
        helpers.assert_close(lse[:H * total].view(H, total)[:, r0:r0 + rows], ref["lse"][:, :rows], f"lse of {b}", atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("B,H", [(3, 2), (60, 8)])   # fewer work items than SMs, and several per SM
@pytest.mark.parametrize("max_len", [128, 400])      # at D = 64 one key tile, and the passes around the main kernel
@pytest.mark.parametrize("D", [64, 128])
def test_backward_writes_inside_the_tensor_only(cuda_device, D, max_len, B, H):
    """Offsets that reach past the tensor at either end, which the host cannot see: no gradient row is written before or behind it.  (All
    tensors lie within larger buffers.)  The sequence that is cut has the gradients of one whose further keys are zeros, as its forward has."""
    spare = 2 * max_len + 100
    lens = [max_len - 38] * (B - 2) + [max_len, max_len]
    cu_list = [0]
    for n in lens:
        cu_list.append(cu_list[-1] + n)
    total = cu_list[-2] - (max_len - 70)   # the last but one has 70 of its rows, the last one begins behind the tensor
    cu = torch.tensor([-40] + cu_list, dtype=torch.int32, device=cuda_device)   # and one before all of them begins before it
    g = torch.Generator(device=cuda_device).manual_seed(7)
    big = [torch.randn(spare + total + spare, H, D, device=cuda_device, generator=g).half() for _ in range(5)]
    q, k, v, d_o, o = (t[spare:spare + total] for t in big)
    status = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    lse = torch.full((spare + H * total + spare,), 7.0, device=cuda_device)
    inside = lse[spare:spare + H * total].view(H, total)
    res = capi.fwd_varlen(q, k, v, cu, max_len, out=o, status=status)
    inside.copy_(res["lse"])
    outs = [torch.full_like(big[0], 7.0) for _ in range(3)]
    grads = [t[spare:spare + total] for t in outs]
    capi.bwd_varlen(d_o, q, k, v, o, inside, cu, max_len, out=tuple(grads), status=status)
    assert capi.check_status(status) == [0, 0, 0, 0]
    for t in outs:
        assert (t[:spare] == 7.0).all() and (t[spare + total:] == 7.0).all() and torch.isfinite(t).all()
    for b in (0, B - 3, B - 2):
        r0, rows = cu_list[b], min(lens[b], total - cu_list[b])
        one = [torch.nn.functional.pad(x[r0:r0 + rows], (0, 0, 0, 0, 0, lens[b] - rows)).permute(1, 0, 2).unsqueeze(0).cpu() for x in (q, k, v, d_o)]
        refs = helpers.composite.attention_grads_fp32(*one, add_mask=None, keep=None, keep_scale=1.0)
        for got, want, name in zip(grads, refs, ("dq", "dk", "dv")):
            helpers.assert_close(got[r0:r0 + rows].permute(1, 0, 2), want[0][:, :rows], f"{name} of {b}")


def test_backward_pass_of_large_and_small_blocks(cuda_device):
    """Head dimension 64: the pass before the main kernel takes blocks of 128 rows on grids of at least 1.5 of them per SM, blocks of 32 below.  The same
    gradients, bit for bit (two key tiles: either order of adding them to dQ's zeros gives the same sum), and zeros in the rows no tile covers."""
    H, D, max_len, tail = 3, 64, 200, 77
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B = (3 * sms + 4 * H - 1) // (4 * H)   # the first batch with 2 * (B * H * 2 blocks of 128 rows) >= 3 * sms
    lens = [(37 * b) % 260 for b in range(B)]   # empty ones, ones past max_len
    q, k, v, d_o, cu = packed_batch(lens + [tail], H, D, torch.float16, seed=9, device=cuda_device)
    got = []
    for n in (B, B - 1):   # the rows behind the last sequence belong to none
        rows = int(cu[n]) + tail if n == B else int(cu[n]) + lens[-1]
        x = [t[:rows] for t in (q, k, v, d_o)]
        res = capi.fwd_varlen(*x[:3], cu[:n + 1].contiguous(), max_len, flags=capi.FLAG_ZERO_UNCOVERED)
        out = tuple(torch.full_like(x[0], float("nan")) for _ in range(3))
        got.append(capi.bwd_varlen(x[3], *x[:3], res["o"], res["lse"], cu[:n + 1].contiguous(), max_len, out=out, flags=capi.FLAG_ZERO_UNCOVERED))
        covered = torch.zeros(rows, dtype=torch.bool, device=cuda_device)
        for b in range(n):
            covered[int(cu[b]):int(cu[b]) + min(lens[b], max_len)] = True
        for t in out:
            assert (t[~covered] == 0).all() and torch.isfinite(t).all()
    end = int(cu[B - 1])
    for large, small in zip(*got):
        assert torch.equal(large[:end], small[:end])


@pytest.mark.parametrize("p", [0.0, 0.2])
@pytest.mark.parametrize("lens,max_len", [([128, 1, 77, 0, 128], 128), ([100, 33, 140, 64], 128), ([20] * 60, 64)])
def test_backward_of_one_key_tile_like_the_padded_batch(cuda_device, lens, max_len, p):
    """Head dimension 64 and up to 128 rows a sequence: one pass zeroes rows, the main kernel does the rest.  The same bits as a sequence on
    its own gives in a padded call (which has no pass at all), zeros in the rows a sequence is cut by and behind the last one."""
    H, D, dtype = 3, 64, torch.float16
    q, k, v, d_o, cu = packed_batch(lens, H, D, dtype, seed=sum(lens), device=cuda_device)
    pad = lambda t: torch.cat([t, torch.ones(9, H, D, dtype=dtype, device=cuda_device)])
    q, k, v, d_o = map(pad, (q, k, v, d_o))
    res = capi.fwd_varlen(q, k, v, cu, max_len, p_drop=p, seed=8, offset=4)
    out = tuple(torch.full_like(q, 7.0) for _ in range(3))
    grads = capi.bwd_varlen(d_o, q, k, v, res["o"], res["lse"], cu, max_len, p_drop=p, seed=8, offset=4, out=out, flags=capi.FLAG_ZERO_UNCOVERED)
    first = cu.tolist()
    for b, n in enumerate(lens):
        n = min(n, max_len)
        if n == 0:
            continue
        rows = slice(first[b], first[b] + n)
        one = [t[rows].transpose(0, 1).unsqueeze(0).contiguous() for t in (d_o, q, k, v, res["o"])]
        lse = res["lse"][:, rows].unsqueeze(0).contiguous()
        kw = dict(p_drop=p, seed=8, offset=4, bh_offset=b * H)
        for got, want in zip(grads, capi.bwd(*one, lse, **kw)):
            assert torch.equal(got[rows], want[0].transpose(0, 1))
        for got in grads:
            assert (got[first[b] + n:first[b + 1]] == 0).all()
    assert all((got[first[-1]:] == 0).all() for got in grads)
