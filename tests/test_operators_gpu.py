"""The operators' host side in C++ (csrc/torch/ops.cpp) against the Python operators that it stands in front of: the same kernels, so the
same bits, launches, gradients and refusals over the layouts that either takes."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def ops(cuda_device):
    from llmctl_b200.ops import functional, native
    native.lib()
    assert not isinstance(native.fast, native._NoOps)
    return functional


@contextlib.contextmanager
def python_operators():
    from llmctl_b200.ops import native
    # what the extension has counted so far stays in launch_count
    fast, native.fast = native.fast, native._NoOps()
    native.count_launches(fast.launches())
    try:
        yield
    finally:
        native.fast = fast
        native.count_launches(-fast.launches())


def _same(a, b):
    if isinstance(a, (tuple, list)):
        assert len(a) == len(b)
        for x, y in zip(a, b):
            _same(x, y)
    else:
        assert a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b)


def _both(run):
    """``run()`` (which makes its own inputs) on either side: outputs and launches."""
    from llmctl_b200.ops import native
    n = native.launch_count
    got = run()
    n = native.launch_count - n
    with python_operators():
        m = native.launch_count
        want = run()
        m = native.launch_count - m
    _same(got, want)
    assert n == m
    return got


def _randn(*shape, seed=0, shift=0):
    """bf16 normals; ``shift``: elements past a 16-byte boundary."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = 1
    for s in shape:
        n *= s
    return torch.randn(n + shift, device="cuda", generator=g).bfloat16()[shift:].view(*shape)


@pytest.mark.parametrize("shape", [(1, 64), (37, 768), (2, 5, 2048), (64,)])
@pytest.mark.parametrize("form", ["plain", "residual", "strided", "odd"])
@pytest.mark.parametrize("grad", [False, True])
def test_rmsnorm(ops, shape, form, grad):
    if form == "odd" and shape != (37, 768):
        pytest.skip("one size is enough")

    def run():
        odd = 1 if form == "odd" else 0
        x = _randn(*shape, shift=odd)
        if form == "strided":
            x = torch.stack([x, x], -1)[..., 0]
        r = _randn(*shape, seed=1, shift=odd) if form != "plain" else None
        w = (1 + _randn(shape[-1], seed=2)).requires_grad_(grad)
        leaves = [w]
        for t in (x, r):
            if t is not None and grad:
                leaves.append(t.requires_grad_(True))
        y, h = ops.rmsnorm(x, w, 1e-5, r)
        assert r is not None or h is x
        if not grad:
            assert not y.requires_grad
            return y, h
        dy, dh = _randn(*shape, seed=3, shift=odd), _randn(*shape, seed=4, shift=odd)
        outs, grads = ((y, h), (dy, dh)) if r is not None else ((y,), (dy,))
        one = torch.autograd.grad(y, leaves, dy, retain_graph=True)        # the other output's gradient is missing
        return (y.detach(), h.detach(), *one, *torch.autograd.grad(outs, leaves, grads))
    _both(run)


@pytest.mark.parametrize("layer", [False, True])
@pytest.mark.parametrize("odd", ["x", "residual", "w", "b", "dy", "dh"])
def test_norms_at_odd_addresses(ops, layer, odd):
    """Operands and gradients that begin inside a 16-byte unit are copied: the same bits as from whole units, on either side."""
    if odd == "b" and not layer:
        pytest.skip("no bias")

    def run(odd):
        def t(name, *shape, seed):
            v, at = _randn(*shape, seed=seed), 1 if name == odd else 0
            return torch.empty(v.numel() + 1, device="cuda", dtype=v.dtype)[at:][:v.numel()].view(shape).copy_(v).requires_grad_(name not in ("dy", "dh"))
        leaves = [t("x", 37, 768, seed=0), t("residual", 37, 768, seed=1), t("w", 768, seed=2)] + ([t("b", 768, seed=3)] if layer else [])
        if layer:
            y, h = ops.layernorm(leaves[0], leaves[2], leaves[3], residual=leaves[1])
        else:
            y, h = ops.rmsnorm(leaves[0], leaves[2], residual=leaves[1])
        return (y.detach(), h.detach(), *torch.autograd.grad((y, h), leaves, (t("dy", 37, 768, seed=4), t("dh", 37, 768, seed=5))))
    _same(_both(lambda: run(odd)), run(""))


@pytest.mark.parametrize("shape,n", [((1, 64), 8), ((32, 256), 64), ((33, 256), 64), ((2, 50, 128), 24), ((300, 72), 40), ((2, 3, 64), 20)])
@pytest.mark.parametrize("form", ["plain", "columns", "odd", "transposed"])
@pytest.mark.parametrize("grad", [False, True])
def test_linear(ops, shape, n, form, grad):
    def run():
        K = shape[-1]
        if form == "columns":
            x = _randn(*shape[:-1], 2 * K)[..., K:]
        elif form == "transposed":
            x = _randn(K, *shape[:-1]).movedim(0, -1)
        else:
            x = _randn(*shape, shift=1 if form == "odd" else 0)
        w = _randn(n, K, seed=1).requires_grad_(grad)
        x = x.detach().requires_grad_(grad)
        y = ops.linear(x, w)
        if not grad:
            return y
        return (y.detach(), *torch.autograd.grad(y, (x, w), _randn(*y.shape, seed=2)))
    _both(run)


def test_linear_makes_the_decode_workspace_where_it_runs(ops, monkeypatch):
    """Calls that the decode GEMM does not take ask for none of its memory."""
    monkeypatch.setattr(ops, "_skinny_ws", {})
    x, w = _randn(4, 64), _randn(48, 64, seed=1)
    ops.linear(x.float(), w.float())
    ops.linear(_randn(40, 64), w)
    ops.linear(x, w.detach().requires_grad_(True))
    ops.linear(x, _randn(48, 64, shift=1))
    assert not ops._skinny_ws
    ops.linear(x, w)
    assert len(ops._skinny_ws) == 1


@pytest.mark.parametrize("rows,width,ffn", [(1, 64, 64), (32, 128, 64), (33, 128, 64), (200, 1024, 256), (130, 256, 96)])
@pytest.mark.parametrize("grad", [False, True])
def test_mlp(ops, rows, width, ffn, grad):
    def run():
        x, up, down = _randn(rows, width), _randn(2 * ffn, width, seed=1), _randn(width, ffn, seed=2)
        leaves = [t.requires_grad_(grad) for t in (x, up, down)]
        y = ops.swiglu_mlp(*leaves)
        return (y.detach(), *torch.autograd.grad(y, leaves, _randn(rows, width, seed=3))) if grad else y
    _both(run)


@pytest.mark.parametrize("form", ["odd", "gaps", "odd gradient"])
@pytest.mark.parametrize("op", ["swiglu", "swiglu_linear", "linear_swiglu", "linear", "mlp"])
def test_gated_layers_on_other_layouts(ops, op, form):
    """Inputs and gradients that begin inside a 16-byte unit, and rows with gaps between them, against whole units back to back: the same bits, and
    nothing is written outside of the gradient."""
    rows, width = 50, 128
    down, up = _randn(64, width // 2, seed=1), _randn(width, width, seed=2)
    w = {"swiglu_linear": [down], "linear_swiglu": [up], "linear": [up], "mlp": [up, _randn(1024, width // 2, seed=3)]}.get(op, [])
    call = {"swiglu": ops.swiglu, "swiglu_linear": ops.swiglu_linear, "linear_swiglu": ops.linear_swiglu, "linear": ops.linear, "mlp": ops.swiglu_mlp}[op]

    def laid_out(t, how):
        if how == "odd":
            return torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:].view(t.shape).copy_(t)
        return torch.cat([t, t], 1)[:, :t.shape[1]] if how == "gaps" else t

    def run(form):
        leaves = [laid_out(_randn(rows, width), form).detach().requires_grad_(True)] + [t.detach().requires_grad_(True) for t in w]
        y = call(*leaves)
        grads = torch.autograd.grad(y, leaves, laid_out(_randn(*y.shape, seed=4), "odd" if form == "odd gradient" else ""))
        return (y.detach(), *grads)
    got, want = run(form), run("")
    if form == "odd" and op in ("linear", "linear_swiglu", "mlp", "swiglu_linear"):         # products of such inputs are the library's
        for a, b in zip(got, want):
            assert (a.float() - b.float()).norm() <= 2.0 ** -7 * b.float().norm()
    else:
        _same(got, want)


@pytest.mark.parametrize("B,S,H,D", [(1, 1, 1, 64), (2, 128, 3, 128), (2, 77, 2, 64), (1, 300, 2, 128)])
@pytest.mark.parametrize("form", ["packed", "apart", "odd", "heads first", "fp32"])
@pytest.mark.parametrize("grad", [False, True])
def test_attention(ops, B, S, H, D, form, grad):
    if form in ("fp32", "heads first") and grad:
        pytest.skip("the library's, whose gradients differ from run to run")
    def run():
        if form == "packed":
            q, k, v = _randn(B, S, 3, H, D).unbind(2)
        elif form == "heads first":
            q, k, v = (_randn(B, H, S, D, seed=i).transpose(1, 2) for i in range(3))
        else:
            q, k, v = (_randn(B, S, H, D, seed=i, shift=1 if form == "odd" and i == 1 else 0) for i in range(3))
        if form == "fp32":
            q, k, v = q.float(), k.float(), v.float()
        leaves = [t.detach().requires_grad_(grad) for t in (q, k, v)]
        o = ops.attention(*leaves, causal=True)
        return (o.detach(), *torch.autograd.grad(o, leaves, _randn(B, S, H, D, seed=5).to(o.dtype))) if grad else o
    _both(run)


@pytest.mark.parametrize("B,S,H,D", [(1, 1, 1, 64), (2, 128, 3, 128), (2, 77, 2, 64)])
@pytest.mark.parametrize("form", ["plain", "positions", "odd", "leaf"])
@pytest.mark.parametrize("grad", [False, True])
def test_rope_attention(ops, B, S, H, D, form, grad):
    from llmctl_b200.ops.attention import rope_attention_packed
    cos, sin = ops.rope_tables(D, 2 * S, device="cuda")

    def run():
        leaf = _randn(B * S, 3 * H * D, shift=1 if form == "odd" else 0).requires_grad_(grad)
        x = leaf if form == "leaf" else torch.empty(B * S * 3 * H * D + 8, dtype=torch.bfloat16, device="cuda")[(1 if form == "odd" else 0):][:leaf.numel()].view_as(leaf).copy_(leaf)
        p = torch.randperm(2 * S, generator=torch.Generator().manual_seed(1))[:S].repeat(B).cuda() if form == "positions" else None
        before = x._version
        o = rope_attention_packed(x, cos, sin, B, S, H, D, positions=p)
        if grad:
            return (o.detach(), *torch.autograd.grad(o, leaf, _randn(B * S, H * D, seed=5)))
        assert (x._version > before) == (form != "odd")                    # rotated in place, and autograd is told; a copy where it cannot be
        return o, x
    _both(run)


@pytest.mark.parametrize("B,H,D,context", [(1, 12, 64, 300), (3, 4, 128, 70), (16, 8, 128, 900)])
def test_paged_decode(ops, B, H, D, context):
    from llmctl_b200.ops import serving

    def run():
        pages = (context + 15) // 16
        k, v = _randn(B * pages, 16, H, D, seed=1), _randn(B * pages, 16, H, D, seed=2)
        tables = torch.randperm(B * pages, generator=torch.Generator().manual_seed(3)).view(B, pages).int().cuda()
        lens = torch.tensor([max(1, context - 13 * i) for i in range(B)], dtype=torch.int32, device="cuda")
        at = lens.long() - 1
        slots = tables.gather(1, (at // 16)[:, None])[:, 0].long() * 16 + at % 16
        slots[B // 2] = -1 if B > 1 else slots[B // 2]
        qkv = _randn(B, 3 * H * D)
        serving.kv_append(qkv, k, v, slots, H, D)
        return serving.paged_attention_decode(qkv[:, :H * D].reshape(B, H, D), k, v, tables, lens, context), k, v
    _both(run)


def _cache_call(B=3, H=2, D=64):
    """Arguments of an append and of a decode over three sequences."""
    k, v = _randn(3 * B, 16, H, D, seed=1), _randn(3 * B, 16, H, D, seed=2)
    tables = torch.randperm(3 * B, generator=torch.Generator().manual_seed(3)).view(B, 3).int().cuda()
    lens = torch.tensor([40, 7, 17], dtype=torch.int32, device="cuda")
    slots = torch.tensor([5, -1, 40], device="cuda")
    return {"qkv": _randn(B, 3 * H * D), "k": k, "v": v, "slots": slots, "tables": tables, "lens": lens, "q": _randn(B, H, D, seed=4)}


def _at_odd_address(t):
    return torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("name,form", [
    ("qkv", _at_odd_address), ("qkv", lambda t: t.t().contiguous().t()), ("slots", lambda t: torch.stack([t, t], 1)[:, 0]), ("slots", lambda t: t.repeat(2)),
    ("qkv", lambda t: torch.cat([t, t], 1)), ("q", _at_odd_address), ("q", lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)), ("q", lambda t: t.transpose(0, 1).contiguous().transpose(0, 1)),
    ("tables", lambda t: torch.cat([t, t], 1)[:, :3]), ("tables", lambda t: t.t().contiguous().t()), ("tables", lambda t: t.repeat(2, 1)), ("lens", lambda t: torch.stack([t, t], 1)[:, 0])])
def test_cache_operators_copy_other_layouts(ops, name, form):
    """Views that the kernels do not read where they lie give what their copies give."""
    from llmctl_b200.ops import serving

    def run(form):
        c = _cache_call()
        c[name] = form(c[name])
        serving.kv_append(c["qkv"], c["k"], c["v"], c["slots"], 2, 64)
        return serving.paged_attention_decode(c["q"], c["k"], c["v"], c["tables"], c["lens"], 48), c["k"], c["v"]
    _same(_both(lambda: run(form)), run(lambda t: t))


@pytest.mark.parametrize("name,form", [
    ("qkv", lambda t: t[:, :383]), ("qkv", lambda t: t.float()), ("k", _at_odd_address), ("v", lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)), ("k", lambda t: t.cpu()),
    ("k", lambda t: t.float()), ("slots", lambda t: t[:2]), ("slots", lambda t: t.int()), ("slots", lambda t: t.cpu())])
def test_append_refuses_what_it_cannot_write(ops, name, form):
    from llmctl_b200.ops import serving
    c = _cache_call()
    c[name] = form(c[name])
    for operators in (contextlib.nullcontext, python_operators):
        with operators(), pytest.raises(ValueError):
            serving.kv_append(c["qkv"], c["k"], c["v"], c["slots"], 2, 64)


@pytest.mark.parametrize("name,form", [
    ("q", lambda t: t.half()), ("k", _at_odd_address), ("v", lambda t: t[:4]), ("v", lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)), ("k", lambda t: t.cpu()), ("k", lambda t: t.half()),
    ("tables", lambda t: t[:2]), ("tables", lambda t: t.long()), ("tables", lambda t: t.cpu()), ("lens", lambda t: t[:2]), ("lens", lambda t: t.long()), ("lens", lambda t: t.cpu())])
def test_decode_refuses_what_it_cannot_read(ops, name, form):
    from llmctl_b200.ops import serving
    c = _cache_call()
    c[name] = form(c[name])
    for operators in (contextlib.nullcontext, python_operators):
        with operators(), pytest.raises(ValueError):
            serving.paged_attention_decode(c["q"], c["k"], c["v"], c["tables"], c["lens"], 48)


def test_saved_tensor_hooks_see_what_is_kept(ops):
    """Offloading and checkpointing pack what a backward will need and unpack it there."""
    packed, unpacked = [], []

    def pack(t):
        packed.append(t)
        return len(packed) - 1

    def unpack(i):
        unpacked.append(i)
        return packed[i]
    q, k, v = (_randn(1, 130, 2, 64, seed=i).requires_grad_(True) for i in range(3))
    w = (1 + _randn(64, seed=4)).requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        y, _ = ops.rmsnorm(ops.attention(q, k, v), w)
    assert len(packed) >= 8
    y.sum().backward()
    assert sorted(unpacked) == list(range(len(packed))) and q.grad.abs().sum() > 0


@pytest.mark.parametrize("form", ["fp32", "cpu", "columns", "part"])
@pytest.mark.parametrize("call", ["linear", "mlp", "two products", "attention"])
def test_saved_tensors_that_come_back_in_other_forms_are_refused(ops, form, call):
    """A hook may give back anything: what the kernels would read wrongly, or out of range, is an error before any launch."""
    def unpack(t):
        return {"fp32": t.float, "cpu": t.cpu, "columns": lambda: t.transpose(0, 1).contiguous().transpose(0, 1), "part": lambda: t[:-1]}[form]()
    x, up, down = (_randn(*size, seed=i).requires_grad_(True) for i, size in enumerate([(40, 64), (256, 64), (64 if call == "two products" else 4096, 128)]))
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        if call == "attention":
            y = ops.attention(*(_randn(2, 130, 2, 64, seed=i).requires_grad_(True) for i in range(3)))
        else:
            y = ops.linear(x, up) if call == "linear" else ops.swiglu_mlp(x, up, down)
    with pytest.raises(RuntimeError):
        y.sum().backward()
    torch.cuda.synchronize()


@pytest.mark.parametrize("form", ["fp32", "cpu", "part", "gaps", "reversed"])
@pytest.mark.parametrize("call", ["norm", "sum and norm", "layer norm", "rotated attention", "rotated attention at positions", "rotation", "gated"])
@pytest.mark.parametrize("extension", [True, False])
def test_saved_tensors_of_norms_and_rotations(ops, extension, call, form):
    """Other types, devices and sizes are an error before any launch, other layouts are copied: the same gradients."""
    from llmctl_b200.ops import attention as attn
    cos, sin = (torch.rand(256, 32, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)) for i in range(2))
    at = torch.arange(130, device="cuda", dtype=torch.int32) + 5

    def spread(t):            # a copy whose numbers lie two apart, or in the other order of the dimensions
        if form == "gaps":
            return torch.stack([t, t], -1)[..., 0]
        return t.permute(*reversed(range(t.dim()))).contiguous().permute(*reversed(range(t.dim())))

    def run(unpack):
        x, r, w, b = (_randn(*z, seed=i).requires_grad_(True) for i, z in enumerate([(130, 384), (130, 384), (384,), (384,)]))
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            y = {"norm": lambda: ops.rmsnorm(x, w)[0], "sum and norm": lambda: ops.rmsnorm(x, w, residual=r)[0], "layer norm": lambda: ops.layernorm(x, w, b)[0],
                 "rotated attention": lambda: attn.rope_attention_packed(x * 1, cos, sin, 1, 130, 2, 64),
                 "rotated attention at positions": lambda: attn.rope_attention_packed(x * 1, cos, sin, 1, 130, 2, 64, at),
                 "rotation": lambda: ops.rope_packed(x * 1, cos, sin, 4, 64, 130), "gated": lambda: ops.swiglu(x)}[call]()
        y.backward(_randn(*y.shape, seed=9))
        return [t.grad for t in (x, r, w, b) if t.grad is not None]
    with contextlib.nullcontext() if extension else python_operators():
        if form in ("gaps", "reversed"):
            _same(run(spread), run(lambda t: t))
        else:
            other = {"fp32": lambda t: t.double() if t.dtype == torch.float32 else t.float(), "cpu": torch.Tensor.cpu, "part": lambda t: t[:-1]}[form]
            with pytest.raises(RuntimeError):
                run(lambda t: other(t) if t.is_cuda and t.is_floating_point() else t)
    torch.cuda.synchronize()


@pytest.mark.parametrize("extension", [True, False])
@pytest.mark.parametrize("call", ["linear", "mlp", "two products"])
def test_saved_rows_that_come_back_with_gaps_give_the_same_gradients(ops, extension, call):
    """The layout that a hook may change without being refused: rows of whole 16-byte units with something between them."""
    def run(unpack):
        leaves = [_randn(*size, seed=i).requires_grad_(True) for i, size in enumerate([(40, 64), (256, 64), (64 if call == "two products" else 4096, 128)])]
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            y = ops.linear(*leaves[:2]) if call == "linear" else ops.swiglu_mlp(*leaves)
        y.backward(_randn(*y.shape, seed=4))
        return [t.grad for t in leaves[:2 if call == "linear" else 3]]
    with contextlib.nullcontext() if extension else python_operators():
        _same(run(lambda t: torch.cat([t, t[:, :8]], 1)[:, :t.shape[1]]), run(lambda t: t))


@pytest.mark.parametrize("wants", ["first", "others", "all"])
@pytest.mark.parametrize("call", ["linear", "mlp", "two products", "attention", "rotated", "norm"])
def test_compiled_autograd(ops, call, wants):
    """A backward that is traced (and run as it was traced, for two lengths) makes the gradients that the engine makes."""
    import torch._dynamo.compiled_autograd as compiled
    from llmctl_b200.ops import attention as attn
    cos, sin = (torch.randn(256, 32, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)) for i in range(2))

    def run(rows, traced):
        sizes = {"linear": [(rows, 64), (128, 64)], "mlp": [(rows, 64), (256, 64), (1024, 128)], "two products": [(rows, 64), (256, 64), (64, 128)],
                 "attention": [(1, rows, 2, 64)] * 3, "rotated": [(rows, 64), (384, 64)], "norm": [(rows, 64), (64,)]}[call]
        leaves = [_randn(*z, seed=i).requires_grad_(wants == "all" or (wants == "first") == (i == 0)) for i, z in enumerate(sizes)]
        y = {"linear": ops.linear, "mlp": ops.swiglu_mlp, "two products": ops.swiglu_mlp, "attention": attn.attention, "norm": lambda x, w: ops.rmsnorm(x, w)[0],
             "rotated": lambda x, w: attn.rope_attention_packed(ops.linear(x, w), cos, sin, 1, rows, 2, 64)}[call](*leaves)
        with compiled._enable(lambda graph: torch.compile(graph, backend="eager")) if traced else contextlib.nullcontext():
            y.backward(_randn(*y.shape, seed=7))
        return [t.grad for t in leaves if t.requires_grad]
    torch._dynamo.reset()
    for rows in (40, 40, 130):
        _same(run(rows, True), run(rows, False))


def test_compiled_autograd_of_weights_with_gradient_buffers(ops):
    """A traced backward leaves the gradient in the weight's buffer and tells its owner, as the engine's does."""
    import torch._dynamo.compiled_autograd as compiled

    def run(traced):
        x, w, told = _randn(130, 64).requires_grad_(True), torch.nn.Parameter(_randn(64, 64, seed=1)), []
        w.main_grad, w._main_grad_fresh, w._grad_ready_cb = torch.ones(w.shape, device="cuda"), False, lambda p: told.append(p is w)
        y = ops.linear(x, w)
        with compiled._enable(lambda graph: torch.compile(graph, backend="eager")) if traced else contextlib.nullcontext():
            y.backward(_randn(130, 64, seed=4))
        assert w.grad is None and told == [True]
        return x.grad, w.main_grad
    torch._dynamo.reset()
    _same(run(True), run(False))


def test_transforms_modes_and_subclasses_go_to_the_python_operators(ops):
    """What wants to see the operators or replace their tensors finds the Python ones, which record or refuse it as before."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from llmctl_b200.ops import native
    x, w = _randn(40, 64), _randn(64, seed=1)

    class Mine(torch.Tensor):
        pass

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    assert native.fast.rmsnorm(x, None, w, 1e-5) is not None
    assert native.fast.rmsnorm(x.as_subclass(Mine), None, w, 1e-5) is None
    assert native.fast.rmsnorm(torch.nn.Parameter(x), None, w, 1e-5) is not None
    with Mode():
        assert native.fast.rmsnorm(x, None, w, 1e-5) is None
    with torch.device("cuda"):
        assert native.fast.rmsnorm(x, None, w, 1e-5) is None
    seen = []
    torch.func.grad(lambda t: (seen.append(native.fast.rmsnorm(t, None, w, 1e-5)), t.float().sum())[1])(x)
    torch.vmap(lambda t: (seen.append(native.fast.rmsnorm(t, None, w, 1e-5)), t)[1])(x)
    torch.vmap(lambda t: (seen.append(native.fast.rmsnorm(x, None, w, 1e-5)), t)[1])(x)
    with torch.autograd.forward_ad.dual_level():
        seen.append(native.fast.rmsnorm(torch.autograd.forward_ad.make_dual(x, x), None, w, 1e-5))
    assert seen == [None] * 4
    with torch.inference_mode():
        y, _ = ops.rmsnorm(x, w)
        assert y.is_inference()
    for bad in (x.float(), x.cpu(), x.half(), x.t(), x[:, :32], 3, None):
        assert native.fast.rmsnorm(bad, None, w, 1e-5) is None


def test_errors_are_the_python_operators_errors(ops):
    """A call that the kernel library refuses raises NativeError from the forward; a wait that ran out is raised before the next launch, in a
    forward and in a backward."""
    from llmctl_b200.ops import native
    x = _randn(40, 12).requires_grad_(True)                                # 12 columns: not whole 16-byte units
    for grad in (False, True):
        with torch.set_grad_enabled(grad), pytest.raises(native.NativeError):
            ops.rmsnorm(x, _randn(12, seed=1))
    x, w = _randn(40, 64).requires_grad_(True), _randn(64, seed=1)
    y, _ = ops.rmsnorm(x, w)
    native.register_signature("llmctl_wait_status_report", [native.c_int, native.c_void_p])

    def run_out():
        assert native.lib().llmctl_wait_status_report(0, native.stream_ptr()) == 0
        torch.cuda.synchronize()
    run_out()
    with pytest.raises(native.NativeError, match="flash attention forward"):
        ops.rmsnorm(x, w)
    run_out()
    with pytest.raises(native.NativeError, match="flash attention forward"):
        torch.autograd.grad(y, x, torch.ones_like(y), retain_graph=True)
    torch.autograd.grad(y, x, torch.ones_like(y))


def test_layers_run_on_several_threads_and_streams(ops):
    """Forward and backward of a few operators on four threads, each on its own stream, against one thread's."""
    import threading
    def run(seed):
        x, w = _randn(300, 128, seed=seed).requires_grad_(True), _randn(384, 128, seed=1)
        y, _ = ops.rmsnorm(x, _randn(128, seed=2))
        o = ops.attention(*ops.linear(y, w).view(1, 300, 3, 2, 64).unbind(2))
        return o.detach(), torch.autograd.grad(o, x, _randn(*o.shape, seed=3))[0]
    want = [run(i) for i in range(4)]
    torch.cuda.synchronize()
    got = [None] * 4

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                got[i] = run(i)
            s.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    _same(got, want)


def test_decode_products_on_several_threads_and_streams(ops):
    """Products of few rows on four threads, each on its own stream, against one thread's: each stream has partials and tickets of its own."""
    import threading
    ws = [_randn(n, 4096, seed=100 + n) for n in (264, 1000)]
    xs = [_randn(5, 4096, seed=i) for i in range(4)]
    want = [[ops.linear(x, w) for w in ws] for x in xs]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            outs = [ops.linear(xs[i], w) for _ in range(100) for w in ws]
            s.synchronize()
            bad.extend(n for n, o in enumerate(outs) if not torch.equal(o, want[i][n % 2]))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_captured_decode_products_replay_beside_others(ops):
    """Two graphs of products of few rows, captured one after the other, replayed on two streams at once and beside products on a third."""
    ws = [_randn(n, 4096, seed=100 + n) for n in (264, 1000)]
    xs = [_randn(5, 4096, seed=i) for i in range(3)]
    want = [[ops.linear(x, w) for w in ws] for x in xs]
    torch.cuda.synchronize()
    graphs, outs = [], []
    for x in xs[:2]:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append([ops.linear(x, w) for _ in range(8) for w in ws])
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in range(3)]
    for _ in range(20):
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(streams[2]):
            eager = [ops.linear(xs[2], w) for _ in range(8) for w in ws]
    torch.cuda.synchronize()
    for got, exact in zip([*outs, eager], want):
        for n, o in enumerate(got):
            assert torch.equal(o, exact[n % 2])


@pytest.mark.parametrize("norm", ["rmsnorm", "layernorm"])
def test_captured_norm_backwards_replay_beside_others(ops, norm):
    """Two captured backwards, replayed on two streams at once: the weights' partial sums of each lie in memory of its own."""
    ins = [(_randn(600, 768, seed=i), (1 + _randn(768, seed=10)), _randn(600, 768, seed=20 + i)) for i in range(2)]

    def run(x, w, dy):
        x, w = x.detach().requires_grad_(True), w.detach().requires_grad_(True)
        return torch.autograd.grad(getattr(ops, norm)(x, w)[0], (x, w), dy)
    want = [run(*i) for i in ins]
    torch.cuda.synchronize()
    graphs, outs = [], []
    for i in ins:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append([run(*i) for _ in range(8)])
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in graphs]
    for _ in range(10):
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
    torch.cuda.synchronize()
    for got, exact in zip(outs, want):
        for o in got:
            _same(o, exact)


def test_capture(ops):
    """A captured layer replays with new inputs."""
    x, w = _randn(64, 128), _randn(384, 128, seed=1)
    n = 1 + _randn(128, seed=2)
    cos, sin = ops.rope_tables(64, 64, device="cuda")
    from llmctl_b200.ops.attention import rope_attention_packed

    def layer(t):
        with torch.no_grad():
            return rope_attention_packed(ops.linear(ops.rmsnorm(t, n)[0], w), cos, sin, 1, 64, 2, 64)
    layer(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = layer(x)
    x.copy_(_randn(64, 128, seed=9))
    g.replay()
    assert torch.equal(out, layer(x))


@pytest.mark.parametrize("rows,width,heads", [(1, 128, 2), (33, 256, 2), (700, 768, 12)])
def test_kernels_begin_when_those_before_have_ended(ops, rows, width, heads):
    """A chain of operators whose kernels are launched beside the end of the one before (csrc/common/dependent.cuh), some of them in place or over
    memory that the one before has just let go of, against the same chain with the device waited for after each."""
    from llmctl_b200.ops import serving
    from llmctl_b200.ops.attention import rope_attention_packed
    D = width // heads
    cos, sin = ops.rope_tables(D, rows, device="cuda")
    n, qkv, out, up, down = (1 + _randn(width, seed=1), _randn(3 * width, width, seed=2) * width ** -0.5, _randn(width, width, seed=3) * width ** -0.5,
                             _randn(4 * width, width, seed=4) * width ** -0.5, _randn(width, 2 * width, seed=5) * width ** -0.5)

    def chain(wait):
        def then(*t):
            if wait:
                torch.cuda.synchronize()
            return t if len(t) > 1 else t[0]
        x, r = _randn(rows, width), _randn(rows, width, seed=6)
        k, v = (torch.zeros(rows, 16, heads, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        tables = torch.arange(rows, device="cuda", dtype=torch.int32).view(rows, 1)
        with torch.no_grad():
            for i in range(12):
                y, r = then(*ops.rmsnorm(x, n, residual=r))
                p = then(ops.linear(y, qkv))
                if D in (64, 128):
                    serving.kv_append(p, k, v, torch.arange(rows, device="cuda") * 16 + i, heads, D)
                    then(k)
                    y = then(serving.paged_attention_decode(p[:, :width].reshape(rows, heads, D), k, v, tables, torch.full((rows,), i + 1, device="cuda", dtype=torch.int32), 16))
                    y = then(ops.linear(y.reshape(rows, width), out))
                    y, r = then(*ops.rmsnorm(y, n, residual=r))
                    p = then(ops.linear(y, qkv))
                y = then(ops.linear(then(rope_attention_packed(p, cos, sin, 1, rows, heads, D)), out))
                y, r = then(*ops.rmsnorm(y, n, residual=r))
                x = then(ops.swiglu_mlp(y, up, down))
        leaves = [t.detach().requires_grad_(True) for t in (x, n, qkv, out, up, down)]
        x = leaves[0]
        y, r = ops.rmsnorm(x, leaves[1])
        o = ops.linear(rope_attention_packed(ops.linear(y, leaves[2]), cos, sin, 1, rows, heads, D), leaves[3])
        y, r = ops.rmsnorm(o, leaves[1], residual=x)
        y = ops.swiglu_mlp(y, leaves[4], leaves[5])
        return (y.detach(), k, v, *torch.autograd.grad((y, r), leaves, (_randn(rows, width, seed=7), _randn(rows, width, seed=8))))
    want = chain(True)
    for _ in range(3):
        _same(chain(False), want)


@contextlib.contextmanager
def waiting_operators():
    """Every kernel of the library is waited for before the next one is launched."""
    from llmctl_b200.ops import native
    call = native.call

    def call_and_wait(*args):
        call(*args)
        torch.cuda.synchronize()
    native.call = call_and_wait
    try:
        with python_operators():
            yield
    finally:
        native.call = call


# prompts: cache write, keys and values rebuilt, attention over them; decoding: cache write, attention in splits and their merge, or in one piece
@pytest.mark.parametrize("starts,tokens,heads", [([0, 0], 300, 4), ([130], 200, 4), ([700, 333, 64], 1, 16), ([2000], 1, 32), ([5, 40], 1, 16)])
def test_latent_kernels_begin_when_those_before_have_ended(ops, starts, tokens, heads):
    """Latent-attention layers one after the other over one cache, whose kernels are launched beside the end of the one before, against the same
    with each kernel waited for."""
    from llmctl_b200.models.mixers import LatentAttention, LatentAttentionSpec
    from llmctl_b200.serve.ragged import Portion, RaggedBatch
    R, dr, dn, dv, page, Q, W = 512, 64, 128, 128, 64, 256, 512
    spec = LatentAttentionSpec(heads=heads, dim=dn, rot_dim=dr, vdim=dv, kv_rank=R, q_rank=Q, scale=(dn + dr) ** -0.5, rot_base=10000.0)
    layers = []
    for i in range(2):
        layers.append(LatentAttention(W, spec, 1e-5, torch.bfloat16, "cuda"))
        with torch.no_grad():
            for j, (name, w) in enumerate(layers[i].named_parameters()):
                w.copy_(_randn(*w.shape, seed=10 * i + j) * (1.0 if w.dim() == 1 else 2 * w.shape[-1] ** -0.5))
    pages = [(s + tokens + page - 1) // page for s in starts]
    tables = [list(range(sum(pages[:i]), sum(pages[:i + 1]))) for i in range(len(starts))]
    batch = RaggedBatch([Portion(i, [1] * tokens, s, [tokens - 1], t) for i, (s, t) in enumerate(zip(starts, tables))], page, torch.device("cuda"))

    def run():
        h = _randn(len(starts) * tokens, W, seed=1)
        caches = [_randn(sum(pages), page, R + dr, seed=2 + i) for i in range(2)]
        with torch.no_grad():
            for i in range(8):
                h = layers[i % 2](h, batch, caches[i % 2])
                h = ops.rmsnorm(h, layers[0].kv_norm)[0]           # 512 weights: the width of the layer
        return h, *caches
    with waiting_operators():
        want = run()
    assert all(t.isfinite().all() for t in want)
    for _ in range(3):
        _same(run(), want)


@pytest.mark.parametrize("rows,V", [(40, 64), (300, 32000), (1100, 4096)])
def test_loss_kernels_begin_when_those_before_have_ended(ops, rows, V):
    """The product before a loss, the loss's three kernels and the gradients behind it, several times over the same memory, as above."""
    w, t = _randn(V, 128, seed=1) * 0.1, torch.randint(0, V, (rows,), generator=torch.Generator().manual_seed(2)).cuda()
    t[::7] = -100

    def run():
        x, out = _randn(rows, 128), []
        for _ in range(6):
            x, leaf = x.detach().requires_grad_(True), w.detach().requires_grad_(True)
            loss = ops.cross_entropy(ops.linear(x, leaf), t, assume_unit_grad=True)
            dx, dw = torch.autograd.grad(loss, (x, leaf))
            out += [loss.detach(), dx, dw]
            x = x.detach() - dx * rows
        return out
    with waiting_operators():
        want = run()
    for _ in range(3):
        _same(run(), want)


@pytest.mark.parametrize("wants", ["x", "w", "up", "down", "x w up down"])
@pytest.mark.parametrize("width", [128, 1024])          # two nodes for the gated layer, one
def test_products_make_the_gradients_that_are_asked_for(ops, wants, width):
    """linear and the gated layer with some of their inputs recorded; a second pass through a graph that is given up is refused."""
    def run():
        t = {"x": _randn(130, 64), "w": _randn(64, 64, seed=1), "up": _randn(192, 64, seed=2), "down": _randn(width, 96, seed=3)}
        wanted = [t[n].requires_grad_(True) for n in wants.split()]
        y = ops.swiglu_mlp(ops.linear(t["x"], t["w"]), t["up"], t["down"])
        dy = _randn(130, width, seed=4)
        first = torch.autograd.grad(y, wanted, dy, retain_graph=True)
        again = torch.autograd.grad(y, wanted, dy)
        _same(first, again)
        with pytest.raises(RuntimeError):
            torch.autograd.grad(y, wanted, dy)
        return (y.detach(), *first)
    _both(run)


def test_weights_with_gradient_buffers(ops):
    """A buffer that is there when the backward runs takes the gradient, fresh or added to, and its owner is told; it need not be there before."""
    def run():
        x, told = _randn(130, 64).requires_grad_(True), []
        ws = [_randn(64, 64, seed=1), _randn(256, 64, seed=2), _randn(1024, 128, seed=3)]
        ws = [torch.nn.Parameter(w) for w in ws]
        y = ops.swiglu_mlp(ops.linear(x, ws[0]), ws[1], ws[2])
        for i, w in enumerate(ws):
            w.main_grad = torch.ones(w.shape, device="cuda")
            w._main_grad_fresh = i == 1
            w._grad_ready_cb = lambda p: told.append([p is w for w in ws].index(True))
        y.backward(_randn(130, 1024, seed=4))
        assert all(w.grad is None for w in ws) and told == [2, 1, 0] and not any(w._main_grad_fresh for w in ws)
        return (x.grad, *(w.main_grad for w in ws))
    _both(run)


@pytest.mark.parametrize("call", ["linear", "mlp", "two products"])
def test_owners_of_gradient_buffers_run_as_anywhere(ops, call):
    """What is told of a finished gradient may update tensors in place, which their versions show, and record a graph."""
    leaves = [torch.nn.Parameter(_randn(*z, seed=i)) for i, z in enumerate([(130, 64), (256, 64), (64 if call == "two products" else 1024, 128)])]
    seen = []

    def told(p):
        t, before = torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda", requires_grad=True)
        t.add_(1)
        with torch.enable_grad():
            seen.append((t._version, (before * 2).requires_grad))
    for w in leaves[1:]:
        w.main_grad, w._grad_ready_cb = torch.zeros(w.shape, device="cuda"), told
    y = ops.linear(*leaves[:2]) if call == "linear" else ops.swiglu_mlp(*leaves)
    y.backward(_randn(*y.shape, seed=4))
    assert seen == [(1, True)] * (1 if call == "linear" else 2)


@pytest.mark.parametrize("B,S,heads,dim", [(1, 33, 2, 64), (2, 130, 2, 128), (1, 600, 12, 64)])
@pytest.mark.parametrize("form", ["plain", "first", "positions", "hook", "few"])
def test_block_without_gradients(ops, B, S, heads, dim, form):
    """A decoder layer as one call against the operators that it is made of; a layer whose parts are watched, or of few rows, is not taken."""
    from llmctl_b200.models.config import ModelConfig
    from llmctl_b200.models.gpt import GPTModel
    from llmctl_b200.ops import native
    S = 20 if form == "few" else S
    B = 1 if form == "few" else B
    torch.manual_seed(1)
    W = heads * dim
    m = GPTModel(ModelConfig(name="t", layers=1, hidden=W, ffn=2 * W, heads=heads, head_dim=dim, vocab_size=128, max_position_embeddings=1024), device="cuda")
    blk, (cos, sin) = m.blocks[0], m.rope_tables(torch.device("cuda"))
    x, r = _randn(B * S, W), None if form == "first" else _randn(B * S, W, seed=1)
    positions = torch.arange(B * S, device="cuda") % S + 3 if form == "positions" else None
    seen, calls = [], []
    if form == "hook":
        blk.attn.out.register_forward_hook(lambda *a: seen.append(1))
    block = native.fast.block

    class Counted:
        def __getattr__(self, name):
            return (lambda *a: (calls.append(1), block(*a))[1]) if name == "block" else getattr(fast, name)
    fast, native.fast = native.fast, Counted()
    try:
        with torch.no_grad():
            got = blk(x, r, cos, sin, B, S, positions)
    finally:
        native.fast = fast
    assert len(calls) == (form not in ("hook", "few"))
    with python_operators(), torch.no_grad():
        want = blk(x, r, cos, sin, B, S, positions)
    _same(got, want)
    assert len(seen) == (2 if form == "hook" else 0)


@pytest.mark.parametrize("dim", [64, 128])
def test_block_holds_no_more_than_its_operators(ops, dim):
    """The most memory that a layer holds as one call, and layer by layer through the extension."""
    from llmctl_b200.models.config import ModelConfig
    from llmctl_b200.models.gpt import GPTModel
    heads = 1024 // dim
    m = GPTModel(ModelConfig(name="t", layers=1, hidden=1024, ffn=1024, heads=heads, head_dim=dim, vocab_size=128, max_position_embeddings=4096), device="cuda")
    blk, (cos, sin) = m.blocks[0], m.rope_tables(torch.device("cuda"))
    x, r = _randn(4096, 1024), _randn(4096, 1024, seed=1)

    def most():
        with torch.no_grad():
            blk(x, r, cos, sin, 1, 4096)
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            y = blk(x, r, cos, sin, 1, 4096)
        torch.cuda.synchronize()
        del y
        return torch.cuda.max_memory_allocated() - before
    whole = most()
    blk._plain = lambda: False
    assert whole <= most()


@pytest.mark.parametrize("starts,width,heads,q_rank,parts", [([0], 256, 16, 128, {}), ([500, 77, 64], 256, 32, 128, {"sink": True}), ([130, 900], 256, 5, 0, {}),
                                                          ([300, 40], 128, 40, 64, {"head_gate": True, "window": 100}), ([70], 128, 8, 64, {"out_gate": True})])
def test_latent_layer_decodes(ops, starts, width, heads, q_rank, parts):
    """A decoding latent-attention layer through the extension against the Python operators around the same kernels."""
    from llmctl_b200.models.mixers import LatentAttention, LatentAttentionSpec
    from llmctl_b200.serve.ragged import Portion, RaggedBatch
    torch.manual_seed(len(starts))
    spec = LatentAttentionSpec(heads=heads, dim=32, rot_dim=64, vdim=24, kv_rank=128, q_rank=q_rank, scale=0.1, rot_base=10000.0, **parts)
    layer = LatentAttention(width, spec, 1e-5, torch.bfloat16, "cuda")
    with torch.no_grad():
        for name, p in layer.named_parameters():
            p.copy_(torch.randn(p.shape, device="cuda") * (0.1 if p.dim() > 1 else 1.0))
    pages = [(s + 64) // 64 for s in starts]
    tables = [list(range(sum(pages[:i]), sum(pages[:i + 1]))) for i in range(len(starts))]
    h, rows = _randn(len(starts), width), _randn(sum(pages), 64, 192, seed=1)

    def run():
        cache = rows.clone()
        batch = RaggedBatch([Portion(i, [0], s, [0], t) for i, (s, t) in enumerate(zip(starts, tables))], 64, torch.device("cuda"))
        with torch.no_grad():
            return layer(h, batch, cache), cache
    with python_operators():
        want = run()
    _same(run(), want)
