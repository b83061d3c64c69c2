"""Shape-only (Meta) kernels of the torch operators: what fake-tensor tracing needs.  Runs without a GPU.

The reference registers its three operators for the CUDA key only (fmha/fmha_manual.cpp:1240-1250 of
shmsong/NvFuserExamples) and has no backward; the Meta kernels and the autograd operator are additions."""
import pytest
import torch


@pytest.fixture(scope="module")
def ops():
    import mha_manual  # noqa: F401  (registers torch.ops.mha_manual)
    return torch.ops.mha_manual


def meta(*shape, dtype=torch.float16):
    return torch.empty(*shape, dtype=dtype, device="meta")


def test_legacy_ops_infer_shapes(ops):
    q, k, v = meta(512, 128, 64), meta(512, 128, 64), meta(512, 128, 64)
    m = meta(512, 128, 128)
    assert ops.fmha_nvfuser(q, k, v, m).shape == (512, 128, 64)
    assert ops.fmha_train_nvfuser(q, k, v, m, m).shape == (512, 128, 64)
    outs = ops.fmha_train_saveim_nvfuser(q, k, v, m, m)
    assert [tuple(o.shape) for o in outs] == [(512, 128, 64), (512, 128, 128), (512, 128, 128)]
    assert all(o.device.type == "meta" and o.dtype == torch.float16 for o in outs)


def test_forward_backward_infer_shapes(ops):
    q, k, v = meta(2, 4, 200, 128, dtype=torch.bfloat16), meta(2, 4, 77, 128, dtype=torch.bfloat16), meta(2, 4, 77, 128, dtype=torch.bfloat16)
    lens = torch.empty(2, dtype=torch.int32, device="meta")
    o, lse = ops.fmha_fwd(q, k, v, None, lens, 0.1, 5, 9)
    assert o.shape == q.shape and o.dtype == torch.bfloat16
    assert lse.shape == (2, 4, 200) and lse.dtype == torch.float32
    dq, dk, dv = ops.fmha_bwd(torch.empty_like(o), q, k, v, o, lse, None, lens, 0.1, 5, 9)
    assert dq.shape == q.shape and dk.shape == k.shape and dv.shape == v.shape
    # [B*H, S, D] inputs give a [B*H, S] logsumexp
    o3, lse3 = ops.fmha_fwd(meta(6, 50, 64), meta(6, 40, 64), meta(6, 40, 64))
    assert o3.shape == (6, 50, 64) and lse3.shape == (6, 50)


def test_autograd_operator_traces_on_meta_tensors(ops):
    q = meta(2, 3, 64, 64).requires_grad_()
    k = meta(2, 3, 96, 64).requires_grad_()
    v = meta(2, 3, 96, 64).requires_grad_()
    o = ops.fmha(q, k, v, None, None, 0.0, 0, 0)
    assert o.shape == q.shape and o.requires_grad
    gq, gk, gv = torch.autograd.grad(o, (q, k, v), torch.empty_like(o))
    assert gq.shape == q.shape and gk.shape == k.shape and gv.shape == v.shape


def test_packed_batch_operators_infer_shapes(ops):
    q, k, v = meta(1000, 4, 64), meta(1000, 4, 64), meta(1000, 4, 64)
    cu = torch.empty(9, dtype=torch.int32, device="meta")
    o, lse = ops.fmha_varlen_fwd(q, k, v, cu, 384, 0.1, 1, 2)
    assert o.shape == (1000, 4, 64) and lse.shape == (4, 1000) and lse.dtype == torch.float32
    dq, dk, dv = ops.fmha_varlen_bwd(torch.empty_like(o), q, k, v, o, lse, cu, 384, 0.1, 1, 2)
    assert dq.shape == dk.shape == dv.shape == (1000, 4, 64)
    qg = meta(1000, 4, 64).requires_grad_()
    out = ops.fmha_varlen(qg, k, v, cu, 384)
    (g,) = torch.autograd.grad(out, (qg,), torch.empty_like(out))
    assert g.shape == qg.shape
    with pytest.raises(RuntimeError, match="same \\[total_rows, H, D\\] shape"):
        ops.fmha_varlen_fwd(q, meta(999, 4, 64), v, cu, 384)


def test_shape_errors_are_raised_without_a_device(ops):
    with pytest.raises(RuntimeError, match="head dimension"):
        ops.fmha_fwd(meta(1, 1, 16, 32), meta(1, 1, 16, 32), meta(1, 1, 16, 32))
    with pytest.raises(RuntimeError, match="sequence lengths differ"):
        ops.fmha_fwd(meta(1, 1, 16, 64), meta(1, 1, 16, 64), meta(1, 1, 24, 64))
    with pytest.raises(RuntimeError, match="float16 or bfloat16"):
        ops.fmha_fwd(meta(1, 1, 16, 64, dtype=torch.float32), meta(1, 1, 16, 64, dtype=torch.float32), meta(1, 1, 16, 64, dtype=torch.float32))
    with pytest.raises(RuntimeError, match="B\\*H\\*S_q\\*S_k"):
        ops.fmha_nvfuser(meta(4, 16, 64), meta(4, 16, 64), meta(4, 16, 64), meta(4, 16, 8))


def test_fused_projection_layout_operators_infer_shapes(ops):
    qkv = meta(2, 300, 3, 4, 64)
    lens = torch.empty(2, dtype=torch.int32, device="meta")
    o, lse = ops.fmha_qkvpacked_fwd(qkv, None, lens, 0.1, 1, 2)
    assert o.shape == (2, 300, 4, 64) and lse.shape == (2, 4, 300) and lse.dtype == torch.float32
    assert ops.fmha_qkvpacked_bwd(torch.empty_like(o), qkv, o, lse, None, lens, 0.1, 1, 2).shape == qkv.shape
    qg = meta(2, 300, 3, 4, 64).requires_grad_()
    out = ops.fmha_qkvpacked(qg, None, lens, 0.1, 1, 2)
    (g,) = torch.autograd.grad(out, (qg,), torch.empty_like(out))
    assert out.shape == (2, 300, 4, 64) and g.shape == qg.shape
    with pytest.raises(RuntimeError):
        ops.fmha_qkvpacked_fwd(meta(2, 300, 2, 4, 64))


def test_packed_fused_projection_operators_infer_shapes(ops):
    qkv = meta(1000, 3, 4, 128, dtype=torch.bfloat16)
    cu = torch.empty(9, dtype=torch.int32, device="meta")
    o, lse = ops.fmha_varlen_qkvpacked_fwd(qkv, cu, 384, 0.1, 1, 2)
    assert o.shape == (1000, 4, 128) and lse.shape == (4, 1000) and lse.dtype == torch.float32
    assert ops.fmha_varlen_qkvpacked_bwd(torch.empty_like(o), qkv, o, lse, cu, 384, 0.1, 1, 2).shape == qkv.shape
    qg = meta(1000, 3, 4, 128, dtype=torch.bfloat16).requires_grad_()
    out = ops.fmha_varlen_qkvpacked(qg, cu, 384)
    (g,) = torch.autograd.grad(out, (qg,), torch.empty_like(out))
    assert g.shape == qg.shape


def test_differentiable_operators_run_below_the_autograd_keys(ops):
    """torch.inference_mode() excludes the autograd keys; the four differentiable operators then reach kernels of their
    own (forward only) instead of failing with "could not run ... with arguments from the 'Meta' backend"."""
    q, k, v = meta(2, 3, 64, 64), meta(2, 3, 96, 64), meta(2, 3, 96, 64)
    cu = torch.empty(5, dtype=torch.int32, device="meta")
    with torch.inference_mode():
        assert ops.fmha(q, k, v).shape == (2, 3, 64, 64)
        assert ops.fmha_qkvpacked(meta(2, 96, 3, 4, 64)).shape == (2, 96, 4, 64)
        assert ops.fmha_varlen(meta(100, 4, 64), meta(100, 4, 64), meta(100, 4, 64), cu, 64).shape == (100, 4, 64)
        assert ops.fmha_varlen_qkvpacked(meta(100, 3, 4, 64), cu, 64).shape == (100, 4, 64)


def test_torch_compile_traces_the_operator_as_one_graph(ops):
    """fullgraph=True: no graph break at the operator, and the compiled backward yields the three gradients."""
    def f(q, k, v):
        return ops.fmha(q * 1.0, k, v, None, None, 0.1, 7, 2, None) * 2.0

    cf = torch.compile(f, fullgraph=True, backend="aot_eager")
    q, k, v = meta(2, 3, 64, 64).requires_grad_(), meta(2, 3, 96, 64).requires_grad_(), meta(2, 3, 96, 64).requires_grad_()
    o = cf(q, k, v)
    assert o.shape == q.shape and o.requires_grad
    gq, gk, gv = torch.autograd.grad(o, (q, k, v), torch.empty_like(o))
    assert gq.shape == q.shape and gk.shape == k.shape and gv.shape == v.shape


def every_differentiable_operator(ops):
    """(call, operands) of the four: `call` takes the operands and keyword arguments."""
    cu = torch.tensor([0, 16, 32], dtype=torch.int32, device="meta")
    qkv = [meta(2, 3, 16, 64) for _ in range(3)]
    return [(ops.fmha, qkv), (ops.fmha_qkvpacked, [meta(2, 16, 3, 4, 64)]),
            (lambda q, k, v, **kw: ops.fmha_varlen(q, k, v, cu, 16, **kw), [meta(32, 3, 64) for _ in range(3)]),
            (lambda qkv, **kw: ops.fmha_varlen_qkvpacked(qkv, cu, 16, **kw), [meta(32, 3, 4, 64)])]


def test_function_transforms_are_refused(ops):
    for call, x in every_differentiable_operator(ops):
        for transform in (lambda f: torch.func.grad(lambda t: f(t).sum())(x[0]), lambda f: torch.func.vjp(f, x[0]),
                          lambda f: torch.func.jvp(f, (x[0],), (x[0],))):
            with pytest.raises(RuntimeError, match="functorch transforms"):
                transform(lambda t: call(t, *x[1:]))


def test_every_tensor_argument_takes_part_in_autograd(ops):
    """A forward-mode tangent is refused on the mask and the lengths as on the operands; an argument that requires a
    gradient, if only the mask, gives an output that does (the mask's own gradient is undefined)."""
    import torch.autograd.forward_ad as fw

    qkv = [meta(2, 3, 16, 64) for _ in range(3)]
    mask, lens = meta(2, 16, dtype=torch.float32), meta(2, dtype=torch.float32)
    with fw.dual_level():
        for args in ((fw.make_dual(qkv[0], meta(2, 3, 16, 64)), *qkv[1:], mask), (*qkv, fw.make_dual(mask, torch.empty_like(mask))),
                     (*qkv, None, fw.make_dual(lens, torch.empty_like(lens)))):
            with pytest.raises(RuntimeError, match="forward-mode"):
                ops.fmha(*args)
    for args in ((*qkv, mask.requires_grad_()), (*qkv, None, lens.requires_grad_())):
        o = ops.fmha(*args)
        assert o.requires_grad
        assert torch.autograd.grad(o, [t for t in args if t is not None and t.requires_grad], torch.empty_like(o), allow_unused=True) == (None,)


def test_backward_runs_under_compiled_autograd(ops):
    from torch._dynamo import compiled_autograd

    graphs = []
    for call, x in every_differentiable_operator(ops):
        x = [t.requires_grad_() for t in x]
        with compiled_autograd._enable(lambda graph: graphs.append(graph) or graph):
            call(*x, p_drop=0.1, scale=0.5, offset_tensor=torch.zeros(1, dtype=torch.int64, device="meta")).sum().backward()
        assert all(t.grad.shape == t.shape for t in x)
    assert len(graphs) == 4


def test_saved_tensor_hooks_run_with_autograd_in_reach(ops):
    """The hooks see the operands, o, lse, the mask and the offset, and what they compute may be differentiable: they run
    outside the region below the autograd keys in which the kernels are called."""
    packed, unpacked = [], []

    def pack(t):
        packed.append(tuple(t.shape))
        return t

    def unpack(t):
        with torch.enable_grad():
            unpacked.append((tuple(t.shape), (torch.zeros(1, requires_grad=True) * 2).requires_grad))
        return t

    q, k, v = (meta(2, 3, 16, 64).requires_grad_() for _ in range(3))
    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        o = ops.fmha(q, k, v, meta(2, 16, dtype=torch.float32), None, 0.1, 1, 2, None, torch.zeros(1, dtype=torch.int64, device="meta"))
    torch.autograd.backward(o, torch.empty_like(o))
    assert packed == 4 * [(2, 3, 16, 64)] + [(2, 3, 16), (2, 16), (1,)]
    assert unpacked == [(shape, True) for shape in packed]
