"""Numerics of every hand-written sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _close(a, b, atol, rtol, what=""):
    a, b = a.float(), b.float()
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    bad = (err > tol)
    assert not bad.any(), (f"{what}: {int(bad.sum())}/{bad.numel()} mismatches, max err {err.max().item():.4g}, "
                           f"first at {torch.nonzero(bad)[0].tolist()}")


@pytest.mark.parametrize("rows,cols", [(64, 768), (4096, 4096), (1000, 5120), (33, 2048)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_fwd_bwd(cuda_device, rows, cols, with_res):
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(0)
    x = torch.randn(rows, cols, device=cuda_device, dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(rows, cols, device=cuda_device, dtype=torch.bfloat16, requires_grad=True) if with_res else None
    w = (1 + 0.1 * torch.randn(cols, device=cuda_device)).to(torch.bfloat16).requires_grad_(True)
    y, h = ops.rmsnorm(x, w, 1e-5, r)
    dy = torch.randn_like(y)
    dh = torch.randn_like(y)
    (y.float() * dy.float()).sum().add((h.float() * dh.float()).sum()).backward()
    # fp32 reference (same rounding point for h as the kernel: bf16)
    xf = x.detach().float().requires_grad_(True)
    rf = r.detach().float().requires_grad_(True) if with_res else None
    wf = w.detach().float().requires_grad_(True)
    hf = xf if rf is None else (xf + rf)
    hq = hf + (hf.detach().to(torch.bfloat16).float() - hf.detach())   # straight-through bf16 rounding
    yf = hq * torch.rsqrt(hq.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    ((yf * dy.float()).sum() + (hq * dh.float()).sum()).backward()
    _close(y, yf, 2e-2, 2e-2, "y")
    _close(x.grad, xf.grad, 3e-2, 3e-2, "dx")
    if with_res:
        _close(r.grad, rf.grad, 3e-2, 3e-2, "dres")
    _close(w.grad, wf.grad, 0.15 * math.sqrt(rows / 64), 3e-2, "dw")


@pytest.mark.parametrize("rows,cols", [(256, 768), (2048, 4096)])
def test_layernorm_fwd_bwd(cuda_device, rows, cols):
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(1)
    x = torch.randn(rows, cols, device=cuda_device, dtype=torch.bfloat16, requires_grad=True)
    w = (1 + 0.1 * torch.randn(cols, device=cuda_device)).to(torch.bfloat16).requires_grad_(True)
    b = (0.1 * torch.randn(cols, device=cuda_device)).to(torch.bfloat16).requires_grad_(True)
    y, _ = ops.layernorm(x, w, b, 1e-5)
    dy = torch.randn_like(y)
    y.backward(dy)
    xf, wf, bf = (t.detach().float().requires_grad_(True) for t in (x, w, b))
    yf = F.layer_norm(xf, (cols,), wf, bf, 1e-5)
    yf.backward(dy.float())
    _close(y, yf, 2e-2, 2e-2, "y")
    _close(x.grad, xf.grad, 3e-2, 3e-2, "dx")
    _close(w.grad, wf.grad, 0.15 * math.sqrt(rows / 64), 3e-2, "dw")
    _close(b.grad, bf.grad, 0.15 * math.sqrt(rows / 64), 3e-2, "db")


def test_rope_fwd_bwd(cuda_device):
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(2)
    B, S, H, D = 2, 256, 8, 128
    cos, sin = ops.rope_tables(D, S, device=cuda_device)
    x = torch.randn(B * S, 3 * H * D, device=cuda_device, dtype=torch.bfloat16, requires_grad=True)
    y = ops.rope_packed(x, cos, sin, 2 * H, D, S)
    dy = torch.randn_like(y)
    y.backward(dy)
    xf = x.detach().float().requires_grad_(True)
    rot = ops._rope_torch(xf[:, :2 * H * D].reshape(B * S, 2 * H, D), cos, sin, None, S, 1.0).reshape(B * S, -1)
    yf = torch.cat([rot, xf[:, 2 * H * D:]], 1)
    yf.backward(dy.float())
    _close(y, yf, 2e-2, 2e-2, "y")
    _close(x.grad, xf.grad, 2e-2, 2e-2, "dx")


@pytest.mark.parametrize("M,Fd", [(512, 1376), (4096, 11008)])
def test_swiglu_fwd_bwd(cuda_device, M, Fd):
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(3)
    gu = torch.randn(M, 2 * Fd, device=cuda_device, dtype=torch.bfloat16, requires_grad=True)
    y = ops.swiglu(gu)
    dy = torch.randn_like(y)
    y.backward(dy)
    gf = gu.detach().float().requires_grad_(True)
    g, u = gf.chunk(2, -1)
    yf = F.silu(g) * u
    yf.backward(dy.float())
    _close(y, yf, 2e-2, 2e-2, "y")
    _close(gu.grad, gf.grad, 3e-2, 3e-2, "dgu")


@pytest.mark.parametrize("grad_dtype", [torch.bfloat16, torch.float32])
def test_adamw_matches_torch(cuda_device, grad_dtype):
    from llmctl_b200.ops import optim
    torch.manual_seed(4)
    n = 1_000_003
    p0 = torch.randn(n, device=cuda_device)
    master, m, v = p0.clone(), torch.zeros_like(p0), torch.zeros_like(p0)
    out = torch.empty(n, device=cuda_device, dtype=torch.bfloat16)
    ref = torch.nn.Parameter(p0.clone())
    opt = torch.optim.AdamW([ref], lr=1e-3, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    scale = torch.tensor([0.5], device=cuda_device)
    for step in range(1, 4):
        g = torch.randn(n, device=cuda_device).to(grad_dtype)
        optim.adamw_step(master, m, v, g, out, step=step, lr=1e-3, beta1=0.9, beta2=0.95, eps=1e-8,
                         weight_decay=0.1, grad_scale=2.0, scale_dev=scale)
        ref.grad = g.float().clone()       # 2.0 * 0.5 = 1
        opt.step()
    _close(master, ref.detach(), 1e-5, 1e-5, "master")
    _close(out, ref.detach(), 1e-2, 1e-2, "bf16 params")
    # non-finite scale => step skipped
    before = master.clone()
    optim.adamw_step(master, m, v, g, out, step=4, lr=1e-3, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1,
                     scale_dev=torch.tensor([float("nan")], device=cuda_device))
    assert torch.equal(before, master)


def test_sumsq(cuda_device):
    from llmctl_b200.ops import optim
    x = torch.randn(3_000_017, device=cuda_device).to(torch.bfloat16)
    out = torch.zeros(1, device=cuda_device)
    optim.sumsq(x, out)
    optim.sumsq(x, out, accumulate=True)
    ref = 2 * x.float().pow(2).sum()
    assert abs(out.item() - ref.item()) / ref.item() < 1e-4


# both sides of every line of the backward (128 | 256 | 512 | 640 | 1024 threads of 8 columns), fewer and more rows than CTAs
@pytest.mark.parametrize("rows,cols", [(1, 8), (700, 264), (1500, 1024), (601, 1032), (1300, 2048), (150, 2056), (800, 4096), (297, 4104), (600, 5120),
                                       (149, 5128), (5, 8184), (400, 8192)])
@pytest.mark.parametrize("layer,with_res", [(False, True), (False, False), (True, True)])
def test_norm_backward_row_lengths(cuda_device, rows, cols, layer, with_res):
    """Gradients against float64 from the same inputs: dx is rounded to bf16 once (2^-9 a number), the weights' sums are fp32 and rounded
    to bf16 at the end; x + r is rounded to bf16 before the norm, which the reference does too."""
    from llmctl_b200.ops import functional as ops
    g = torch.Generator(device=cuda_device).manual_seed(rows + cols)
    rand = lambda *s: torch.randn(*s, device=cuda_device, generator=g).bfloat16()      # noqa: E731
    x, r, w, b, dy, dh = rand(rows, cols), rand(rows, cols), rand(cols), rand(cols), rand(rows, cols), rand(rows, cols)
    leaves = [t.clone().requires_grad_(True) for t in (x, w, b)]
    res = r if with_res else None
    y, h = ops.layernorm(*leaves, 1e-5, res) if layer else ops.rmsnorm(*leaves[:2], 1e-5, res)
    torch.autograd.backward([y, h] if with_res else [y], [dy, dh] if with_res else [dy])
    want = [t.double().requires_grad_(True) for t in (x + r if with_res else x, w, b)]
    hd = want[0] * 1
    yd = F.layer_norm(hd, (cols,), want[1], want[2], 1e-5) if layer else hd * (hd.pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt() * want[1]
    torch.autograd.backward([yd, hd] if with_res else [yd], [dy.double(), dh.double()] if with_res else [dy.double()])
    for a, e in list(zip(leaves, want))[:3 if layer else 2]:
        bound = 2.0 ** -8 * e.grad.norm()
        if not with_res and rows * cols <= 8:       # dx of one short row is a difference of near numbers: fp32 of its terms
            bound = bound + 2.0 ** -20 * dy.double().norm() * w.double().norm()
        assert (a.grad.double() - e.grad).norm() <= bound


@pytest.mark.parametrize("rows,V", [(128, 32000), (1024, 32768), (64, 4096), (32, 50304)])
def test_cross_entropy(cuda_device, rows, V):
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(5)
    base = (2 * torch.randn(rows, V, device=cuda_device)).to(torch.bfloat16)
    t = torch.randint(0, V, (rows,), device=cuda_device)
    t[::7] = -100
    lin = base.clone().requires_grad_(True)
    logits = lin * 1.0                    # non-leaf, consumed in place
    loss = ops.cross_entropy(logits, t, grad_scale=0.5, assume_unit_grad=True)
    loss.backward()
    lf = base.float().requires_grad_(True)
    lref = 0.5 * F.cross_entropy(lf, t, ignore_index=-100)
    lref.backward()
    assert abs(loss.item() - lref.item()) < 2e-3 * max(1.0, abs(lref.item()))
    _close(lin.grad, lf.grad, 2e-5, 3e-2, "dlogits")


# Both sides of every line of the row kernels (8192 | ring of three rows | of two | streamed), more rows than CTAs
@pytest.mark.parametrize("rows,V", [(300, 8192), (300, 8200), (500, 16384), (149, 16392), (7, 37544), (450, 37552), (150, 56320), (3, 56328)])
def test_cross_entropy_row_lengths(cuda_device, rows, V):
    """Loss and gradient against float64, with masked logits (-inf and the type's lowest value) and ignored targets.  The gradient is
    rounded to bf16 (2^-9); exponentials and sums are fp32."""
    from llmctl_b200.ops import functional as ops, native
    torch.manual_seed(V)
    base = (2 * torch.randn(rows, V, device=cuda_device)).bfloat16()
    base[:, 5:900:7] = float("-inf")
    base[:, 6:900:7] = torch.finfo(torch.bfloat16).min
    base[1, 2:] = torch.finfo(torch.bfloat16).min
    t = torch.randint(900, V, (rows,), device=cuda_device)
    t[::9], t[1], t[2] = -100, 0, V - 1
    leaf = base.clone().requires_grad_(True)
    ops.cross_entropy(leaf * 1.0, t, assume_unit_grad=True).backward()
    assert native.lib().llmctl_cross_entropy_status(1) == 0
    with torch.no_grad():
        plain = ops.cross_entropy(base, t)
    ref = base.double().requires_grad_(True)
    want = F.cross_entropy(ref, t)
    want.backward()
    assert abs(plain.item() - want.item()) <= 1e-5 * want.abs().item()
    assert (leaf.grad.double() - ref.grad).norm() <= 2.0 ** -8.5 * ref.grad.norm()
    assert not leaf.grad[::9].any()


@pytest.mark.parametrize("rows", [0, 1, 31, 1023, 1024, 1025, 9001])
def test_cross_entropy_mean(cuda_device, rows):
    """The mean of the rows' losses: fewer and more rows than the summing block has threads, some or all of them ignored.  A row's loss
    errs by some 4 units of fp32 of its largest terms (below 16 here), a sum of n numbers by no more than log2(1024) + n / 1024 units."""
    from llmctl_b200.ops import functional as ops
    g = torch.Generator(device=cuda_device).manual_seed(rows)
    base = torch.randn(rows, 64, device=cuda_device, generator=g).bfloat16()
    t = torch.randint(0, 64, (rows,), device=cuda_device, generator=g)
    t[::5] = -1
    for targets, scale in ((t, 0.25), (torch.full_like(t, -1), 1.0)):
        leaf = base.clone().requires_grad_(True)
        loss = ops.cross_entropy(leaf * 1.0, targets, ignore_index=-1, grad_scale=scale)
        loss.backward()
        ref = base.double().requires_grad_(True)
        want = scale * F.cross_entropy(ref, targets, ignore_index=-1, reduction="sum") / max(1, int((targets != -1).sum()))
        want.backward()
        assert loss.shape == () and loss.dtype == torch.float32
        assert abs(loss.item() - want.item()) <= 2.0 ** -24 * (4 * 16 + (10 + rows / 1024) * abs(want.item()))
        assert (leaf.grad.double() - ref.grad).norm() <= 2.0 ** -8.5 * ref.grad.norm()


GEMM_SHAPES = [(128, 256, 64), (256, 512, 256), (4096, 4096, 4096), (1000, 2752, 1376), (384, 136, 200),
               (8192, 1024, 512)]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm_layouts(cuda_device, M, N, K, a_mn, b_mn):
    from llmctl_b200.ops import functional as ops
    if (M % 8 and a_mn) or (N % 8):
        pytest.skip("leading dims must be multiples of 8")
    torch.manual_seed(6)
    A = torch.randn(M, K, device=cuda_device).to(torch.bfloat16)
    B = torch.randn(N, K, device=cuda_device).to(torch.bfloat16)
    ref = A.float() @ B.float().t()
    a_arg = A.t().contiguous() if a_mn else A
    b_arg = B.t().contiguous() if b_mn else B
    for tile_n in (128, 192, 256, 2, 3, 0):
        out = ops.gemm_raw(a_arg, b_arg, a_mn=a_mn, b_mn=b_mn, tile_n=tile_n)
        _close(out, ref, 0.05 * math.sqrt(K / 64), 2e-2, f"gemm tile_n={tile_n}")


@pytest.mark.parametrize("M,N,K,splits", [(8, 4096, 4096, 0), (1, 4096, 4096, 4), (16, 12288, 4096, 0), (17, 4096, 11008, 0),
                                            (32, 1000, 512, 3), (5, 32000, 4096, 1), (8, 22016, 4096, 0)])
def test_gemm_skinny(cuda_device, M, N, K, splits):
    """Decode GEMM (swap-AB, split-K with in-kernel deterministic fix-up) vs fp32 matmul; twice in a row so the
    self-resetting ticket counters are exercised, and bit-identical between the two calls."""
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(8)
    x = torch.randn(M, K, device=cuda_device).to(torch.bfloat16)
    w = torch.randn(N, K, device=cuda_device).to(torch.bfloat16)
    ref = x.float() @ w.float().t()
    out1 = ops.gemm_skinny(x, w, splits=splits)
    out2 = ops.gemm_skinny(x, w, splits=splits)
    _close(out1, ref, 0.05 * math.sqrt(K / 64), 2e-2, "skinny gemm")
    assert torch.equal(out1, out2)
    with torch.no_grad():
        assert torch.equal(ops.linear(x, w), out1) or splits != 0


@pytest.mark.parametrize("M,N,K", [(1, 8, 512), (17, 1000, 520), (32, 1536, 4096), (16, 1544, 2048), (5, 4096, 256), (9, 4104, 136), (32, 8192, 128), (15, 8200, 128),
                                   (3, 104, 448), (2, 2048, 64)])
def test_gemm_skinny_clusters(cuda_device, M, N, K):
    """Decode GEMM where a cluster shares a tile's K (eights, fours and pairs to either side of their lines, shares of one block and uneven ones, too
    few blocks for a cluster) against float64: fp32 sums rounded to bf16, 2 x 2^-9 in the 2-norm; equal bits in a second call, and no writes past
    the rows that there are."""
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(N)
    x, w = torch.randn(M, K, device=cuda_device).bfloat16(), torch.randn(N, K, device=cuda_device).bfloat16()
    out = torch.full((M + 1, N), 7.0, device=cuda_device, dtype=torch.bfloat16)
    ops.gemm_skinny(x, w, out=out[:M])
    want = x.double() @ w.double().t()
    assert (out[:M].double() - want).norm() <= 2 * 2.0 ** -9 * want.norm() and (out[M] == 7).all()
    assert torch.equal(ops.gemm_skinny(x, w), out[:M])


def test_gemm_fp32_accumulate(cuda_device):
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(7)
    M, N, K = 512, 768, 1024
    A = torch.randn(M, K, device=cuda_device).to(torch.bfloat16)
    B = torch.randn(N, K, device=cuda_device).to(torch.bfloat16)
    C = torch.randn(M, N, device=cuda_device)
    ref = C + A.float() @ B.float().t()
    ops.gemm_raw(A, B, out=C, accumulate=True)
    _close(C, ref, 1e-2, 1e-3, "fp32 accumulate")
    C2 = torch.randn(M, N, device=cuda_device)
    ref2 = C2 + A.float() @ B.float().t()
    ops.gemm_raw(A, B, out=C2, accumulate=True, tile_n=2)
    _close(C2, ref2, 1e-2, 1e-3, "fp32 accumulate (2-CTA)")


def test_linear_autograd(cuda_device):
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(8)
    x = torch.randn(4, 128, 1024, device=cuda_device).to(torch.bfloat16).requires_grad_(True)
    w = (0.05 * torch.randn(2048, 1024, device=cuda_device)).to(torch.bfloat16).requires_grad_(True)
    y = ops.linear(x, w)
    dy = torch.randn_like(y)
    y.backward(dy)
    xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    yf = F.linear(xf, wf)
    yf.backward(dy.float())
    _close(y, yf, 5e-2, 2e-2, "y")
    _close(x.grad, xf.grad, 5e-2, 2e-2, "dx")
    _close(w.grad, wf.grad, 0.5, 2e-2, "dw")


# One wave of 128 x 64 tiles, of 128 x 128 tiles, and beyond (CTA pairs): both sides of each line of the automatic tile choice on
# 148 SMs, with ragged rows, columns and K, every operand layout and output type.
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (130, 72, 200), (37 * 128, 256, 64), (37 * 128 + 1, 256, 64), (74 * 128 - 3, 256, 72),
                                   (74 * 128 + 8, 256, 72), (776, 2304, 136)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, False), (False, True), (True, True)])
def test_gemm_automatic_tiles(cuda_device, M, N, K, a_mn, b_mn):
    """Against float64; fp32 accumulation of bf16 products: sqrt(K) 2^-24 and the rounding of the output (2^-9 bf16)."""
    from llmctl_b200.ops import functional as ops
    if a_mn and M % 8:
        M = M + 8 - M % 8          # the row pitch of a [K, M] operand is whole 16-byte units
    torch.manual_seed(M + N)
    a = torch.randn(K, M, device=cuda_device).bfloat16() if a_mn else torch.randn(M, K, device=cuda_device).bfloat16()
    b = torch.randn(K, N, device=cuda_device).bfloat16() if b_mn else torch.randn(N, K, device=cuda_device).bfloat16()
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    for dtype, bound in ((torch.bfloat16, 2.0 ** -9), (torch.float32, 2.0 ** -20)):
        pool = torch.full((M + 3, N), 7.0, device=cuda_device, dtype=dtype)
        out = ops.gemm_raw(a, b, a_mn=a_mn, b_mn=b_mn, out=pool[:M])
        assert (out.double() - want).norm() <= bound * want.norm()
        assert bool((pool[M:] == 7).all())
        ops.gemm_raw(a, b, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=True)
        assert (out.double() - 2 * want).norm() <= 2 * bound * (2 * want).norm()


# Rows around the decode GEMM's 32 and the tiles of 128 / 256, gate columns around 64 / 128, both tile kernels, ragged K
@pytest.mark.parametrize("M,F_,K", [(32, 64, 64), (33, 8, 72), (129, 136, 200), (1000, 2048, 768), (300, 5632, 264), (2560, 1032, 128)])
def test_linear_swiglu(cuda_device, M, F_, K):
    """Forward and gradients against float64 of the same bf16 inputs.  Forward: one rounding of the output (the composed path rounds
    gate and up too); backward: gate, up, their gradients and the results are rounded to bf16, 2^-9 each."""
    from llmctl_b200.ops import functional as ops, native
    torch.manual_seed(M)
    x = torch.randn(M, K, device=cuda_device).bfloat16().requires_grad_(True)
    w = (torch.randn(2 * F_, K, device=cuda_device) / K ** 0.5).bfloat16().requires_grad_(True)
    dy = torch.randn(M, F_, device=cuda_device).bfloat16()
    before = native.launch_count
    y = ops.linear_swiglu(x, w)
    assert native.launch_count == before + (1 if M > 32 else 2)
    dx, dw = torch.autograd.grad(y, (x, w), dy)
    with torch.no_grad():
        assert (ops.linear_swiglu(x, w).double() - y.double()).norm() <= 2.0 ** -8 * y.double().norm()
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    g, u = (xd @ wd.t()).chunk(2, -1)
    want = F.silu(g) * u
    gx, gw = torch.autograd.grad(want, (xd, wd), dy.double())
    assert (y.double() - want).norm() <= (2.0 ** -9 if M > 32 else 2.0 ** -7.5) * want.norm()
    assert (dx.double() - gx).norm() <= 2.0 ** -7 * gx.norm() and (dw.double() - gw).norm() <= 2.0 ** -7 * gw.norm()


def test_linear_swiglu_of_extreme_halves(cuda_device):
    """Gates where the sigmoid is 0 beside halves near the largest bf16: 0 as from the separate kernels, not the NaN of inf * 0; products
    that overflow by themselves stay infinite."""
    from llmctl_b200.ops import functional as ops
    x = torch.zeros(64, 64, device=cuda_device).bfloat16()
    x[:, 0] = 1
    gate = torch.tensor([-120.0, -90.0, 0.0, 2.0, 100.0, -3.0, 88.0, 1.0], device=cuda_device)
    up = torch.tensor([3e38, -3e38, 3e38, 1e38, 3e38, 1e38, -2e38, -1.0], device=cuda_device)
    w = torch.zeros(16, 64, device=cuda_device).bfloat16()
    w[:8, 0], w[8:, 0] = gate.bfloat16(), up.bfloat16()
    got = ops.linear_swiglu(x, w)
    want = ops.swiglu(ops.linear(x, w))
    assert torch.equal(got.isinf(), want.isinf()) and not got.isnan().any() and not want.isnan().any()
    fine = ~want.isinf()
    assert torch.allclose(got[fine].double(), want[fine].double(), rtol=2.0 ** -8, atol=0)
    assert (got[:, :2] == 0).all() and got[:, 4].isinf().all()


# One-wave tiles of 64 and 128 columns and the pair tile, rows and columns that end inside a tile, ragged K
@pytest.mark.parametrize("M,F_,K,N", [(33, 8, 64, 72), (200, 136, 264, 64), (1000, 2048, 768, 768), (2560, 1032, 128, 200), (2049, 5632, 64, 320)])
def test_swiglu_mlp(cuda_device, monkeypatch, M, F_, K, N):
    """Forward and gradients against float64 of the same bf16 inputs: the activation, gate, up, their gradients and the results are
    rounded to bf16 (2^-9 each); what the down-projection hands to the activation is not."""
    from llmctl_b200.ops import functional as ops, native
    monkeypatch.setattr(ops, "SWIGLU_BWD_COLS", 0)
    torch.manual_seed(M)
    x = torch.randn(M, K, device=cuda_device).bfloat16().requires_grad_(True)
    w_up = (torch.randn(2 * F_, K, device=cuda_device) / K ** 0.5).bfloat16().requires_grad_(True)
    w_down = (torch.randn(N, F_, device=cuda_device) / F_ ** 0.5).bfloat16().requires_grad_(True)
    dy = torch.randn(M, N, device=cuda_device).bfloat16()
    before = native.launch_count
    y = ops.swiglu_mlp(x, w_up, w_down)
    grads = torch.autograd.grad(y, (x, w_up, w_down), dy)
    assert native.launch_count == before + 6
    composed = ops.linear(ops.linear_swiglu(x, w_up), w_down)
    general = torch.autograd.grad(composed, (x, w_up, w_down), dy)
    assert torch.equal(y, composed)
    xd, ud, dd = (t.detach().double().requires_grad_(True) for t in (x, w_up, w_down))
    g, u = (xd @ ud.t()).chunk(2, -1)
    want = torch.autograd.grad((F.silu(g) * u) @ dd.t(), (xd, ud, dd), dy.double())
    for got, old, ref in zip(grads, general, want):
        err, was = ((t.double() - ref).norm() / ref.norm() for t in (got, old))
        assert err <= 2.0 ** -7 and err <= 1.02 * was, (float(err), float(was))


@pytest.mark.parametrize("B,S,H", [(2, 512, 4), (1, 2048, 2), (3, 128, 1), (1, 1024, 8)])
@pytest.mark.parametrize("packed", [True, False])
def test_flash_attention_fwd(cuda_device, B, S, H, packed):
    """tcgen05 flash attention forward vs fp32 softmax(QK^T/sqrt(d))V with a causal mask."""
    from llmctl_b200.ops import attention as attn, native
    if not native.has_symbol("llmctl_flash_attn_fwd"):
        pytest.skip("flash attention kernel not built")
    D = 128
    torch.manual_seed(9)
    if packed:
        qkv = torch.randn(B, S, 3, H, D, device=cuda_device).bfloat16()
        q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    else:
        q, k, v = (torch.randn(B, S, H, D, device=cuda_device).bfloat16() for _ in range(3))
    assert attn._native_ok(q, k, v)
    with torch.no_grad():
        o = attn.attention(q, k, v, causal=True)
    qf, kf, vf = (t.float().transpose(1, 2) for t in (q, k, v))
    s = qf @ kf.transpose(-1, -2) / math.sqrt(D)
    mask = torch.triu(torch.ones(S, S, dtype=torch.bool, device=cuda_device), 1)
    s = s.masked_fill(mask, float("-inf"))
    ref = (torch.softmax(s, -1) @ vf).transpose(1, 2)
    _close(o, ref, 2e-2, 2e-2, "attention out")
    lse = torch.empty(B, H, S, dtype=torch.float32, device=cuda_device)
    o2 = torch.empty(B, S, H, D, dtype=torch.bfloat16, device=cuda_device)
    native.call("llmctl_flash_attn_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o2.data_ptr(), lse.data_ptr(), B, S, H, D,
                q.stride(1), k.stride(1), v.stride(1), o2.stride(1), 1.0 / math.sqrt(D), 1, native.stream_ptr())
    _close(lse, torch.logsumexp(s, -1), 2e-2, 1e-3, "lse")


@pytest.mark.parametrize("B,S,H", [(2, 256, 2), (1, 1024, 4), (2, 128, 1)])
def test_flash_attention_bwd(cuda_device, B, S, H):
    """tcgen05 flash attention backward (dq, dk, dv) vs autograd through the fp32 reference."""
    from llmctl_b200.ops import attention as attn, native
    if not native.has_symbol("llmctl_flash_attn_bwd"):
        pytest.skip("flash attention backward kernel not built")
    D = 128
    torch.manual_seed(10)
    qkv = (0.5 * torch.randn(B, S, 3, H, D, device=cuda_device)).bfloat16().requires_grad_(True)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    o = attn.attention(q, k, v, causal=True)
    do = torch.randn_like(o)
    o.backward(do)
    ref_in = qkv.detach().float().requires_grad_(True)
    qf, kf, vf = (ref_in[:, :, i].transpose(1, 2) for i in range(3))
    s = qf @ kf.transpose(-1, -2) / math.sqrt(D)
    s = s.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device=cuda_device), 1), float("-inf"))
    ref = (torch.softmax(s, -1) @ vf).transpose(1, 2)
    ref.backward(do.float())
    _close(o, ref, 2e-2, 2e-2, "out")
    for i, name in enumerate(("dq", "dk", "dv")):
        _close(qkv.grad[:, :, i], ref_in.grad[:, :, i], 4e-2, 4e-2, name)


@pytest.mark.parametrize("S", [77, 200, 1000])
def test_flash_attention_ragged_lengths_use_the_native_kernel(cuda_device, S):
    """Causal attention over a length that is not a multiple of the 128-token tile (every serving prefill): padded to
    the tile, run by the tcgen05 kernel (not SDPA), forward and backward vs the fp32 reference."""
    from llmctl_b200.ops import attention as attn, native
    if not native.has_symbol("llmctl_flash_attn_bwd"):
        pytest.skip("flash attention kernels not built")
    B, H, D = 2, 4, 128
    torch.manual_seed(12)
    qkv = (0.5 * torch.randn(B, S, 3, H, D, device=cuda_device)).bfloat16().requires_grad_(True)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    before = native.launch_count
    o = attn.attention(q, k, v, causal=True)
    assert native.launch_count > before, "ragged causal attention fell back to the library path"
    do = torch.randn_like(o)
    o.backward(do)
    ref_in = qkv.detach().float().requires_grad_(True)
    qf, kf, vf = (ref_in[:, :, i].transpose(1, 2) for i in range(3))
    s = qf @ kf.transpose(-1, -2) / math.sqrt(D)
    s = s.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device=cuda_device), 1), float("-inf"))
    ref = (torch.softmax(s, -1) @ vf).transpose(1, 2)
    ref.backward(do.float())
    _close(o, ref, 2e-2, 2e-2, "out")
    for i, name in enumerate(("dq", "dk", "dv")):
        _close(qkv.grad[:, :, i], ref_in.grad[:, :, i], 4e-2, 4e-2, name)


def test_flash_attention_head_dim_64_uses_the_native_kernel(cuda_device):
    """head_dim 64 (gpt-125m) at a ragged length: forward and backward vs the fp32 reference."""
    from llmctl_b200.ops import attention as attn, native
    if not native.has_symbol("llmctl_flash_attn_bwd"):
        pytest.skip("flash attention kernels not built")
    B, S, H, D = 2, 300, 6, 64
    torch.manual_seed(13)
    qkv = (0.5 * torch.randn(B, S, 3, H, D, device=cuda_device)).bfloat16().requires_grad_(True)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    before = native.launch_count
    o = attn.attention(q, k, v, causal=True)
    assert native.launch_count > before and o.shape == (B, S, H, D)
    do = torch.randn_like(o)
    o.backward(do)
    ref_in = qkv.detach().float().requires_grad_(True)
    qf, kf, vf = (ref_in[:, :, i].transpose(1, 2) for i in range(3))
    s = qf @ kf.transpose(-1, -2) / math.sqrt(D)
    s = s.masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool, device=cuda_device), 1), float("-inf"))
    ref = (torch.softmax(s, -1) @ vf).transpose(1, 2)
    ref.backward(do.float())
    _close(o, ref, 2e-2, 2e-2, "out")
    for i, name in enumerate(("dq", "dk", "dv")):
        _close(qkv.grad[:, :, i], ref_in.grad[:, :, i], 4e-2, 4e-2, name)


# K shared by a cluster: every number of CTAs (uneven shares of K and of the 64 columns), one k-block each, ragged tiles, all layouts, two CTAs
# to an SM (100 tiles), and sizes for which it is chosen.
@pytest.mark.parametrize("M,N,K,a_mn,b_mn,splits", [
    (1, 8, 128, 0, 0, 2), (100, 72, 200, 0, 0, 3), (136, 200, 1000, 0, 1, 4), (200, 136, 1000, 1, 0, 5), (128, 64, 448, 1, 1, 7), (264, 72, 4104, 1, 1, 8),
    (640, 1280, 264, 0, 0, 4), (300, 768, 1000, 0, 1, 6), (200, 768, 32000, 0, 1, 0), (64, 2048, 5632, 0, 0, 0), (768, 768, 3000, 1, 1, 0)])
def test_gemm_split_k(cuda_device, M, N, K, a_mn, b_mn, splits):
    """Against float64: fp32 sums of K exact products rounded to bf16 (2^-9 in the 2-norm, and as much again for the sums), and added to
    what fp32 outputs hold (2^-16)."""
    from llmctl_b200.ops import native
    torch.manual_seed(M + N)
    a = torch.randn(K, M, device=cuda_device).bfloat16() if a_mn else torch.randn(M, K, device=cuda_device).bfloat16()
    b = torch.randn(K, N, device=cuda_device).bfloat16() if b_mn else torch.randn(N, K, device=cuda_device).bfloat16()
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())

    def product(out, beta):
        native.call("llmctl_gemm_bf16", a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0), a_mn, b_mn,
                    int(out.dtype == torch.float32), beta, -splits, 0, native.stream_ptr())
        return out.double()
    err = product(torch.full((M, N), float("nan"), device=cuda_device, dtype=torch.bfloat16), 0) - want
    assert err.norm() <= 2 * 2.0 ** -9 * want.norm()
    old = torch.randn(M, N, device=cuda_device)
    err = product(old.clone(), 1) - (want + old)
    assert err.norm() <= 2.0 ** -16 * (want + old).norm()
    old = old.bfloat16()
    err = product(old.clone(), 1) - (want + old)
    assert err.norm() <= 2 * 2.0 ** -9 * (want + old).norm()


@pytest.mark.parametrize("M,N,K,a_mn,b_mn,chosen", [(200, 768, 32000, 0, 1, 4), (64, 2048, 5632, 0, 0, 4), (768, 768, 4000, 1, 1, 2), (500, 768, 32000, 0, 1, 4),
                                                    (768, 768, 3000, 1, 1, 1), (200, 2048, 2048, 0, 0, 1), (500, 2048, 5632, 0, 0, 1)])
def test_gemm_split_k_is_chosen(cuda_device, M, N, K, a_mn, b_mn, chosen):
    """On either side of the rule's line: the bits of the number of CTAs that it gives a tile, whose sums no other order leaves alike."""
    from llmctl_b200.ops import native
    torch.manual_seed(1)
    a = torch.randn(*((K, M) if a_mn else (M, K)), device=cuda_device).bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), device=cuda_device).bfloat16()

    def product(tile):
        out = torch.empty(M, N, device=cuda_device)
        native.call("llmctl_gemm_bf16", a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0), a_mn, b_mn, 1, 0, tile, 0,
                    native.stream_ptr())
        return out
    for splits in (1, 2, 4, 8):
        assert torch.equal(product(0), product(64 if splits == 1 else -splits)) == (splits == chosen), splits


@pytest.mark.parametrize("M,heads,K,seq", [(1, 1, 64, 1), (33, 3, 200, 11), (130, 12, 768, 130), (777, 12, 768, 259), (777, 20, 136, 777), (2000, 12, 72, 500), (4100, 16, 64, 1025)])
@pytest.mark.parametrize("form", ["plain", "positions", "one part"])
def test_gemm_with_rotation(cuda_device, M, heads, K, seq, form):
    """The packed projection with its rotation (one wave of either narrow tile, pair tiles, ragged rows) against the product and the rotation after it:
    the same bits."""
    from llmctl_b200.ops import functional as ops, native
    torch.manual_seed(M)
    N = 3 * heads * 64
    x, w = torch.randn(M, K, device=cuda_device).bfloat16(), torch.randn(N, K, device=cuda_device).bfloat16()
    cos, sin = torch.randn(2048, 32, device=cuda_device), torch.randn(2048, 32, device=cuda_device)
    positions = torch.randint(0, 2048, (M,), device=cuda_device, dtype=torch.int32) if form == "positions" else None
    parts = heads if form == "one part" else 2 * heads
    got = torch.full((M, N), float("nan"), device=cuda_device, dtype=torch.bfloat16)
    native.register_signature("llmctl_gemm_rope_bf16", [native.c_void_p] * 3 + [native.c_int] * 3 + [native.c_ll] * 3 + [native.c_void_p] * 3 + [native.c_int] * 2 + [native.c_void_p])
    native.call("llmctl_gemm_rope_bf16", x.data_ptr(), w.data_ptr(), got.data_ptr(), M, N, K, K, K, N, cos.data_ptr(), sin.data_ptr(), native.ptr(positions), seq,
                parts * 64, native.stream_ptr())
    want = ops.gemm_raw(x, w, tile_n=128)
    native.call("llmctl_rope_inplace", want.data_ptr(), N, M, parts, 64, cos.data_ptr(), sin.data_ptr(), native.ptr(positions), seq, 1.0, native.stream_ptr())
    assert torch.equal(got, want)


# Lengths around the 128-row blocks and the 256-query items, more items than SMs (256 x 3 blocks), several head groups of the
# backward's item order (S = 2048: 16 heads of 128 to a group), non-causal whole blocks, views at an odd address (copied first).
@pytest.mark.parametrize("B,S,H,D,causal,shift", [
    (1, 1, 1, 128, True, 0), (2, 127, 3, 64, True, 0), (1, 128, 2, 64, True, 0), (2, 129, 2, 128, True, 0), (1, 255, 2, 64, True, 0),
    (2, 257, 3, 128, True, 0), (8, 384, 32, 64, True, 0), (1, 2048, 20, 128, True, 0), (2, 256, 2, 64, False, 0), (1, 384, 2, 128, False, 0),
    (2, 200, 2, 128, True, 1), (1, 128, 2, 64, True, 1)])
def test_flash_attention_edges_of_blocks(cuda_device, B, S, H, D, causal, shift):
    """Forward and backward against float64.  Inputs are exact, P, dS and the outputs are rounded to bf16 (2^-9 each): 3 x 2^-9 in
    the 2-norm.  At S = 1 dq and dk are zero up to the rounding of o in delta = dO . O."""
    from llmctl_b200.ops import attention as attn, native
    torch.manual_seed(S)
    flat = torch.randn(B * S * 3 * H * D + shift, device=cuda_device).bfloat16()[shift:].view(B, S, 3, H, D)
    q, k, v = (flat[:, :, i].detach().requires_grad_(True) for i in range(3))
    assert attn._native_ok(q, k, v, causal) == (shift == 0)
    do = torch.randn(B, S, H, D, device=cuda_device).bfloat16()
    before = native.launch_count
    o = attn.attention(q, k, v, causal=causal)
    got = (o.detach(), *torch.autograd.grad(o, (q, k, v), do))
    assert native.launch_count == before + 3
    assert native.lib().llmctl_flash_fwd_status(1) == 0 and native.lib().llmctl_flash_bwd_status(1) == 0
    for h in range(H):          # one head at a time: float64 scores of all heads would not be small
        qd, kd, vd = (t.detach()[:, :, h].double().requires_grad_(True) for t in (q, k, v))
        s = qd @ kd.transpose(-1, -2) / math.sqrt(D)
        if causal:
            s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=cuda_device).triu(1), float("-inf"))
        od = torch.softmax(s, -1) @ vd
        want = (od.detach(), *torch.autograd.grad(od, (qd, kd, vd), do[:, :, h].double()))
        for name, a, b in zip(("o", "dq", "dk", "dv"), got, want):
            a = a[:, :, h].double()
            bound = 3 * 2.0 ** -9 * b.norm() if S > 1 or name in ("o", "dv") else 2.0 ** -8 * do.double().norm() * v.double().norm() * q.double().norm()
            assert (a - b).norm() <= bound, f"{name} head {h}: {((a - b).norm() / b.norm()).item():.2e}"


# Keys split between the two warpgroups: one block and two (the second half has one or none), odd and even counts, a ragged end, more tiles
# than SMs, no mask.
@pytest.mark.parametrize("B,S,H,D,causal", [(1, 129, 2, 64, True), (1, 256, 3, 128, True), (1, 385, 3, 64, True), (2, 600, 2, 128, True), (1, 2000, 12, 64, True),
                                            (1, 1500, 16, 128, True), (1, 640, 2, 64, False), (2, 768, 2, 128, False)])
def test_flash_attention_split_keys(cuda_device, B, S, H, D, causal):
    """Output against float64 (P and the output are rounded to bf16: 2 x 2^-9 in the 2-norm) and the log-sum-exp against float64 sums of exact
    products (fp32 sums of up to S terms and the approximate exponential: 1e-5 of the largest)."""
    from llmctl_b200.ops import attention as attn, native
    torch.manual_seed(S)
    qkv = torch.randn(B, S, 3, H, D, device=cuda_device).bfloat16()
    q, k, v = (qkv[:, :, i] for i in range(3))
    o, lse = torch.empty(B, S, H, D, dtype=torch.bfloat16, device=cuda_device), torch.empty(B, H, S, device=cuda_device)
    native.call("llmctl_flash_attn_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B, S, H, D, q.stride(1), k.stride(1),
                v.stride(1), o.stride(1), 1.0 / math.sqrt(D), int(causal), native.stream_ptr())
    assert native.lib().llmctl_flash_fwd_status(1) == 0
    with torch.no_grad():
        assert torch.equal(attn.attention(q, k, v, causal=causal), o)
    for h in range(H):
        s = q[:, :, h].double() @ k[:, :, h].double().transpose(-1, -2) / math.sqrt(D)
        if causal:
            s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=cuda_device).triu(1), float("-inf"))
        want = torch.softmax(s, -1) @ v[:, :, h].double()
        assert (o[:, :, h].double() - want).norm() <= 2 * 2.0 ** -9 * want.norm()
        exact = torch.logsumexp(s, -1)
        assert (lse[:, h].double() - exact).abs().max() <= 1e-5 * exact.abs().max().clamp(min=1)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("keys", [slice(512, None), slice(0, 512), slice(600, 700)])
def test_flash_attention_scores_of_minus_infinity(cuda_device, D, keys):
    """Keys whose scores are -inf weigh nothing, also where they are all that a row sees of one half of the keys (blocks of 128: 0 to 3 and 4 to 6 of
    the last rows); a row that sees no other has no result.  Bound as above."""
    from llmctl_b200.ops import attention as attn
    torch.manual_seed(1)
    q, k, v = (torch.randn(1, 777, 12, D, device=cuda_device).bfloat16() for _ in range(3))
    q[..., 0] = q[..., 0].abs() + 0.1
    k[:, keys, :, 0] = float("-inf")
    got = attn.attention(q, k, v).double()
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) / math.sqrt(D)
    s = s.masked_fill(torch.ones(777, 777, dtype=torch.bool, device=cuda_device).triu(1), float("-inf"))
    want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v.double())
    assert torch.equal(got.isnan(), want.isnan())
    assert (got - want).nan_to_num().norm() <= 2 * 2.0 ** -9 * want.nan_to_num().norm()


@pytest.mark.parametrize("which", [0, 1, 2])
def test_whole_tiles_at_odd_addresses_are_copied(cuda_device, which):
    """Heads of 128 and whole 128-token tiles where one of q, k and v begins at an odd address: the kernels run on copies, and nothing else
    (the library's attention reads 16-byte units at the address that it is given)."""
    from llmctl_b200.ops import attention as attn, native
    torch.manual_seed(which)
    qkv = [torch.randn(2 * 128 * 3 * 128 + 1, device=cuda_device).bfloat16()[int(i == which):][:2 * 128 * 3 * 128].view(2, 128, 3, 128).detach().requires_grad_(True)
           for i in range(3)]
    do = torch.randn(2, 128, 3, 128, device=cuda_device).bfloat16()
    before = native.launch_count
    o = attn.attention(*qkv)
    got = (o.detach(), *torch.autograd.grad(o, qkv, do))
    assert native.launch_count == before + 3
    whole = [t.detach().clone().requires_grad_(True) for t in qkv]
    o = attn.attention(*whole)
    for a, b in zip(got, (o.detach(), *torch.autograd.grad(o, whole, do))):
        assert torch.equal(a, b)


# several items of one to five blocks per CTA, so that tiles, statistics and accumulators are handed on between items of every length and kind
@pytest.mark.parametrize("B,S,H,D,causal", [(4, 640, 40, 128, True), (4, 520, 70, 64, True), (12, 100, 64, 128, True), (3, 384, 100, 64, False)])
def test_flash_attention_backward_over_many_items(cuda_device, B, S, H, D, causal):
    """Gradients against float64 products of a few heads (bounds as above), and again, bit for bit: nothing depends on who takes which item."""
    from llmctl_b200.ops import attention as attn, native
    torch.manual_seed(S)
    q, k, v = (torch.randn(B, S, H, D, device=cuda_device).bfloat16().requires_grad_(True) for _ in range(3))
    do = torch.randn(B, S, H, D, device=cuda_device).bfloat16()
    o = attn.attention(q, k, v, causal=causal)
    got = torch.autograd.grad(o, (q, k, v), do, retain_graph=True)
    for a, b in zip(got, torch.autograd.grad(o, (q, k, v), do)):
        assert torch.equal(a, b)
    assert native.lib().llmctl_flash_bwd_status(1) == 0
    for h in (0, H // 2, H - 1):
        qd, kd, vd = (t.detach()[:, :, h].double().requires_grad_(True) for t in (q, k, v))
        s = qd @ kd.transpose(-1, -2) / math.sqrt(D)
        if causal:
            s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=cuda_device).triu(1), float("-inf"))
        want = torch.autograd.grad(torch.softmax(s, -1) @ vd, (qd, kd, vd), do[:, :, h].double())
        for name, a, b in zip(("dq", "dk", "dv"), got, want):
            assert (a[:, :, h].double() - b).norm() <= 3 * 2.0 ** -9 * b.norm(), f"{name} head {h}"


@pytest.mark.parametrize("S,D", [(130, 64), (128, 64), (77, 128), (128, 128)])
@pytest.mark.parametrize("packed", [False, True])
def test_flash_attention_gradients_at_odd_addresses(cuda_device, S, D, packed):
    """The incoming gradient is read in 16-byte units: one that begins elsewhere is copied, and the gradients are those of the copy."""
    from llmctl_b200.ops import attention as attn, functional as ops
    torch.manual_seed(S)
    B, H = 2, 3
    flat = torch.randn(B * S * H * D + 1, device=cuda_device).bfloat16()
    odd = flat[1:]
    assert odd.data_ptr() % 16 == 2
    leaf = torch.randn(B * S, 3 * H * D, device=cuda_device).bfloat16().requires_grad_(True)
    cos, sin = ops.rope_tables(D, S, device=cuda_device)
    def grad(do):
        x = leaf * 1
        if packed:
            o = attn.rope_attention_packed(x, cos, sin, B, S, H, D)
        else:
            o = attn.attention(*x.view(B, S, 3, H, D).unbind(2))
        return torch.autograd.grad(o, leaf, do.view(o.shape))[0]
    assert torch.equal(grad(odd), grad(odd.clone()))


def test_flash_backward_of_short_items_beside_other_work(cuda_device):
    """One block per sequence: thousands of the shortest items in a row, while copies on another stream slow the stores of the
    accumulators down.  The gradients are those of an undisturbed run, bit for bit, and no wait runs out."""
    from llmctl_b200.ops import attention as attn, native
    torch.manual_seed(3)
    B, S, H, D = 64, 128, 32, 64
    q, k, v = (torch.randn(B, S, H, D, device=cuda_device).bfloat16().requires_grad_(True) for _ in range(3))
    do = torch.randn(B, S, H, D, device=cuda_device).bfloat16()
    def grads():
        return torch.autograd.grad(attn.attention(q, k, v), (q, k, v), do)
    want = grads()
    side, a = torch.cuda.Stream(), torch.empty(128 << 20, dtype=torch.uint8, device=cuda_device)
    b = torch.empty_like(a)
    torch.cuda.synchronize()
    for _ in range(20):
        with torch.cuda.stream(side):
            for _ in range(4):
                b.copy_(a)
        got = grads()
        assert all(torch.equal(x, y) for x, y in zip(got, want))
    torch.cuda.synchronize()
    assert native.lib().llmctl_flash_fwd_status(1) == 0 and native.lib().llmctl_flash_bwd_status(1) == 0



@pytest.mark.parametrize("M,N,K", [(8, 4096, 1376), (8, 4096, 512), (5, 1000, 200), (32, 2752, 4096), (1, 4096, 1384)])
def test_skinny_gemm_k_tail_and_odd_shapes(cuda_device, M, N, K):
    """Decode GEMM on shapes whose K is not a multiple of the 64-deep k-block (GPT-7B down-projection at TP=8:
    K = 1376) and on N that is not a multiple of the tile: vs fp32 matmul."""
    from llmctl_b200.ops import functional as ops, native
    if not native.has_symbol("llmctl_gemm_skinny_bf16"):
        pytest.skip("skinny GEMM not built")
    torch.manual_seed(0)
    x = torch.randn(M, K, device=cuda_device).bfloat16()
    w = (0.05 * torch.randn(N, K, device=cuda_device)).bfloat16()
    y = ops.gemm_skinny(x, w)
    ref = x.float() @ w.float().t()
    assert ((y.float() - ref).abs().max() / ref.abs().max()).item() < 1e-2


@pytest.mark.parametrize("which", [0, 1, 2, 3])
def test_a_wait_reported_on_the_device_is_raised_on_the_host(cuda_device, which):
    """The byte that a kernel sets when its wait runs out, set by a kernel that does nothing else."""
    from llmctl_b200.ops import native
    native.register_signature("llmctl_wait_status_report", [native.c_int, native.c_void_p])
    native.call("llmctl_wait_status_report", which, native.stream_ptr())
    torch.cuda.synchronize()
    with pytest.raises(native.NativeError, match=native._WAITS[which][0]):
        native.check_waits()
    native.check_waits()


@pytest.mark.parametrize("V", [8192, 8200, 16392, 32000, 40000, 56328])
def test_cross_entropy_of_rows_that_are_not_finite(cuda_device, V):
    """Rows without a finite logit, with an infinite one or with a NaN: NaN in the loss and in the whole row's gradient, on every path (short
    rows in registers, rows in the ring with exponentials kept and without, streamed rows), and nowhere else; parts masked to -inf stay 0."""
    from llmctl_b200.ops import functional as ops
    torch.manual_seed(V)
    inf = float("inf")
    x = torch.randn(9, V, device=cuda_device).bfloat16()
    x[0] = -inf
    x[1, 5] = inf
    x[2, V - 1] = float("nan")
    x[3, : V // 2] = -inf
    x[4, 1:] = -inf
    x[5] = -inf
    x[6, 3:V - 3] = -inf
    t = torch.tensor([0, 7, 9, V - 1, 0, -100, 1, 3, -100], device=cuda_device)
    ref = x.float().requires_grad_(True)
    rows = torch.nn.functional.cross_entropy(ref, t, reduction="none")
    rows.sum().backward()
    for i in range(9):
        leaf = x[i:i + 1].clone().requires_grad_(True)
        loss = ops.cross_entropy(leaf * 1, t[i:i + 1])
        grad = torch.autograd.grad(loss, leaf)[0]
        assert torch.equal(grad.isnan(), ref.grad[i:i + 1].isnan()), i
        assert bool(loss.isnan()) == bool(rows[i].isnan()), i
        if not ref.grad[i].isnan().any():
            assert torch.allclose(grad.float(), ref.grad[i:i + 1], rtol=2.0 ** -7, atol=1e-6), i
            assert torch.allclose(loss, rows[i], rtol=1e-4, atol=1e-5), i
