"""Multi-GPU worker (one process per GPU, launched by torchrun from tests/test_multigpu.py or by hand):
numerics of every fused compute+collective kernel against NCCL + PyTorch, and device-timed comparisons."""
import json
import os
import sys
import tempfile
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))

import torch  # noqa: E402
import torch.distributed as dist  # noqa: E402


def time_max(fn, iters=10, warm=3):
    for _ in range(warm):
        fn()
    dist.barrier(); torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(iters):
        fn()
    e1.record(); torch.cuda.synchronize()
    t = torch.tensor([e0.elapsed_time(e1) / iters], device="cuda")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t)


def cpu_us(fn, iters=20):
    """Host time to enqueue one call (the GPU is drained first, so this is pure launch cost)."""
    import time
    torch.cuda.synchronize(); dist.barrier()
    t0 = time.perf_counter()
    for _ in range(iters):
        fn()
    t = (time.perf_counter() - t0) / iters * 1e6
    torch.cuda.synchronize()
    return t


def case_probe(out):
    from llmctl_b200.comms import symm
    buf = symm.SymmBuffer(1 << 20, torch.bfloat16)
    out["symm"] = {"world": buf.world, "multicast_ptr": hex(buf.multicast_ptr), "signal_pad_bytes": buf.signal_pad_bytes,
                   "p2p": [torch.cuda.can_device_access_peer(buf.rank, r) for r in range(buf.world) if r != buf.rank]}
    buf.tensor.fill_(buf.rank + 1)
    torch.cuda.synchronize(); buf.barrier()
    peer = (buf.rank + 1) % buf.world
    t = buf.handle.get_buffer(peer, (16,), torch.bfloat16)
    out["symm"]["peer_read_ok"] = bool((t == peer + 1).all())
    buf.barrier()


def case_tp_kernels(out, M=4096, K=4096, N=1536, Kl=1376):
    """K1 ag_gemm, K2 gemm_rs (+ reduce + rmsnorm), K11 — numerics vs NCCL + PyTorch and timings."""
    from llmctl_b200.comms import fused
    from llmctl_b200.comms.mesh import init_mesh
    from llmctl_b200.ops import native
    from llmctl_b200.ops.functional import gemm_raw as ops_gemm
    st = init_mesh(tp=dist.get_world_size(), sequence_parallel=True)
    ctx = fused.init_tp_workspace(max_tokens=M, hidden=4096)
    assert ctx is not None, "fused TP context unavailable"
    W, r = st.tp, st.tp_rank
    Ms = M // W
    torch.manual_seed(100 + r)
    x_local = torch.randn(Ms, K, device="cuda").bfloat16()
    w = (0.02 * torch.randn(N, K, device="cuda")).bfloat16()
    # ---- K1 ----
    res = {}
    for it in range(3):                                  # several calls: exercises the alternating buffers / epochs
        y, xg = ctx._ag_gemm_fused(x_local, w)
        gathered = torch.empty(M, K, device="cuda", dtype=torch.bfloat16)
        dist.all_gather_into_tensor(gathered, x_local)
        ref = gathered.float() @ w.float().t()
        err = (y.float() - ref).abs().max().item() / ref.abs().max().item()
        per_chunk = [((y.float() - ref)[c * Ms:(c + 1) * Ms].abs().max() / ref.abs().max()).item() for c in range(W)]
        assert torch.equal(xg, gathered), f"gathered activation mismatch (call {it})"
        assert err < 2e-2, f"ag_gemm rel err {err} on call {it}, per source chunk {per_chunk}"
    res["ag_gemm_rel_err"] = err

    def base_ag():
        g = torch.empty(M, K, device="cuda", dtype=torch.bfloat16)
        dist.all_gather_into_tensor(g, x_local)
        return g @ w.t()
    res["ag_gemm_ms"] = time_max(lambda: ctx._ag_gemm_fused(x_local, w), iters=30)
    res["ag_gemm_enqueue_us"] = cpu_us(lambda: ctx._ag_gemm_fused(x_local, w))
    res["nccl_ag_then_cublas_enqueue_us"] = cpu_us(base_ag)
    # the two halves on their own: push without a consumer, GEMM with every flag already raised
    from llmctl_b200.comms.fused import K1_FLAG_BASE
    buf = ctx.xg[0]
    mine = buf.tensor[:M * K].view(M, K)[r * Ms:(r + 1) * Ms]

    def push_only(ctas, R, mc=True):
        def f():
            ctx.ep_ag += 1
            native.call("llmctl_ag_push", mine.data_ptr(), buf.peers, (buf.multicast_ptr or None) if mc else None, Ms, K, R,
                        buf.pads, K1_FLAG_BASE, r, W, ctx.ep_ag, ctx.push_counters.data_ptr(), 1, ctas, native.stream_ptr())
        return f
    parts = {}
    for ctas in (16, 32, 64, 148):
        for R in sorted({min(256, Ms), Ms}):
            parts[f"push_ctas{ctas}_R{R}_us"] = 1e3 * time_max(push_only(ctas, R), iters=20)
    parts["push_p2p_ctas64_us"] = 1e3 * time_max(push_only(64, min(256, Ms), mc=False), iters=20)
    yy = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)

    def gemm_only():
        native.call("llmctl_gemm_bf16_gated", buf.tensor.data_ptr(), w.data_ptr(), yy.data_ptr(), M, N, K, K, w.stride(0), N,
                    0, 0, 0, 0, 0, buf.signal_ptrs[r] + 4 * K1_FLAG_BASE, 1, min(256, Ms), r, W, native.stream_ptr())
    parts["gated_gemm_flags_set_us"] = 1e3 * time_max(gemm_only, iters=20)
    parts["plain_gemm_native_us"] = 1e3 * time_max(lambda: ops_gemm(gathered, w), iters=20)
    res["k1_parts"] = parts
    sweep = {}
    for tile in (2, 256, 128):
        for slab in sorted({128, 256, Ms}):
            if Ms % slab:
                continue
            ctx.tile_n, ctx.slab_rows = tile, slab
            sweep[f"tile{tile}_slab{slab}"] = time_max(lambda: ctx._ag_gemm_fused(x_local, w), iters=20)
    ctx.tile_n, ctx.slab_rows = 0, 256
    res["ag_gemm_ms_sweep"] = sweep
    ctx.ag_gemm(x_local, w)                    # auto mode: times both paths on this shape once
    res["k1_autotune"] = ctx.path_report()
    # MN-major weight (backward of a row-parallel layer): same product from w^T stored [K, N]
    wt = w.t().contiguous()
    y_mn, _ = ctx._ag_gemm_fused(x_local, wt, w_mn=True)
    assert (y_mn.float() - ref).abs().max().item() / ref.abs().max().item() < 2e-2, "ag_gemm with MN-major weight"
    if ctx.xg[0].multicast_ptr:
        ctx.use_multicast = False
        y_p2p, _ = ctx._ag_gemm_fused(x_local, w)
        assert torch.equal(y_p2p, y), "P2P push differs from the NVLS push"
        res["ag_gemm_p2p_push_ms"] = time_max(lambda: ctx._ag_gemm_fused(x_local, w))
        ctx.use_multicast = True
    res["nccl_ag_then_cublas_ms"] = time_max(base_ag)
    res["gemm_only_cublas_ms"] = time_max(lambda: gathered @ w.t())
    # ---- K2 ----
    torch.manual_seed(200 + r)
    x2 = torch.randn(M, Kl, device="cuda").bfloat16()
    w2 = (0.02 * torch.randn(4096, Kl, device="cuda")).bfloat16()
    resid = torch.randn(Ms, 4096, device="cuda").bfloat16()
    nw = (1 + 0.1 * torch.randn(4096, device="cuda")).bfloat16()
    for it in range(3):
        h, y2, rstd = ctx.gemm_rs(x2, w2, residual=resid, norm_w=nw)
        part = (x2.float() @ w2.float().t()).bfloat16()        # each rank's partial is rounded to bf16 before the sum
        full = part.float().clone()
        dist.all_reduce(full)
        href = (full[r * Ms:(r + 1) * Ms] + resid.float())
        e1 = (h.float() - href).abs().max().item() / href.abs().max().item()
        hq = h.float()
        yref = hq * torch.rsqrt(hq.pow(2).mean(-1, keepdim=True) + 1e-5) * nw.float()
        e2 = (y2.float() - yref).abs().max().item()
        assert e1 < 2e-2 and e2 < 5e-2, f"gemm_rs errs {e1} {e2} on call {it}"
    res["gemm_rs_rel_err"] = e1
    h_mn, _, _ = ctx.gemm_rs(x2, w2.t().contiguous(), residual=resid, w_mn=True)
    assert (h_mn.float() - href).abs().max().item() / href.abs().max().item() < 2e-2, "gemm_rs with MN-major weight"

    def base_rs():
        p = x2 @ w2.t()
        o = torch.empty(Ms, 4096, device="cuda", dtype=torch.bfloat16)
        dist.reduce_scatter_tensor(o, p)
        hh = o + resid
        return torch.nn.functional.rms_norm(hh, (4096,), nw, 1e-5)
    res["gemm_rs_norm_ms"] = time_max(lambda: ctx.gemm_rs(x2, w2, residual=resid, norm_w=nw))
    res["cublas_nccl_rs_norm_ms"] = time_max(base_rs)
    res["gemm_only_cublas_ms_k2"] = time_max(lambda: x2 @ w2.t())
    # ---- K11 ----
    B, H = 8, 4096
    sb = ctx.stage[0]
    for it in range(1, 4):
        part = torch.randn(B, H, device="cuda").bfloat16()
        sb.tensor[:B * H].view(B, H).copy_(part)
        res_in = torch.randn(B, H, device="cuda").bfloat16()
        hout, yout = torch.empty_like(res_in), torch.empty_like(res_in)
        native.call("llmctl_ar_residual_rmsnorm", sb.peers, 0, None, sb.pads, 16, r, W, res_in.data_ptr(), hout.data_ptr(),
                    nw.data_ptr(), yout.data_ptr(), B, H, 1e-5, it, None, 0, native.stream_ptr())
        tot = part.float().clone(); dist.all_reduce(tot)
        hr = (tot + res_in.float())
        assert (hout.float() - hr).abs().max().item() < 0.1, "K11 h mismatch"
        hq = hout.float()
        yr = hq * torch.rsqrt(hq.pow(2).mean(-1, keepdim=True) + 1e-5) * nw.float()
        assert (yout.float() - yr).abs().max().item() < 5e-2, "K11 y mismatch"
        torch.cuda.synchronize(); dist.barrier()
    ep = [10]

    def k11():
        ep[0] += 1
        native.call("llmctl_ar_residual_rmsnorm", sb.peers, 0, None, sb.pads, 16, r, W, res_in.data_ptr(), hout.data_ptr(),
                    nw.data_ptr(), yout.data_ptr(), B, H, 1e-5, ep[0], None, 0, native.stream_ptr())

    def base_k11():
        t = part.clone(); dist.all_reduce(t)
        return torch.nn.functional.rms_norm(t + res_in, (H,), nw, 1e-5)
    res["ar_rmsnorm_us"] = 1e3 * time_max(k11, iters=50)
    res["nccl_ar_add_norm_us"] = 1e3 * time_max(base_k11, iters=50)
    if sb.multicast_ptr:
        def k11mc():
            ep[0] += 1
            native.call("llmctl_ar_residual_rmsnorm", sb.peers, 0, sb.multicast_ptr, sb.pads, 16, r, W, res_in.data_ptr(),
                        hout.data_ptr(), nw.data_ptr(), yout.data_ptr(), B, H, 1e-5, ep[0], None, 0, native.stream_ptr())
        k11mc(); torch.cuda.synchronize()
        assert (hout.float() - hr).abs().max().item() < 0.1, "K11 multimem mismatch"
        res["ar_rmsnorm_multimem_us"] = 1e3 * time_max(k11mc, iters=50)
    # roofline fractions of the fused paths: the slower of compute at the measured bf16 peak and NVLink bytes at the
    # measured link rate, over the achieved time (metrics/roofline.py)
    from llmctl_b200.metrics.roofline import RooflinePoint
    res["roofline"] = {
        "k1_ag_gemm": RooflinePoint("ag_gemm", res["ag_gemm_ms"] * 1e-3, flops=2.0 * M * N * K,
                                    nvlink_bytes=(W - 1) * Ms * K * 2).report(),
        "k2_gemm_rs": RooflinePoint("gemm_rs+reduce+norm", res["gemm_rs_norm_ms"] * 1e-3, flops=2.0 * M * 4096 * Kl,
                                    nvlink_bytes=(W - 1) * Ms * 4096 * 2).report(),
        "k11_ar_rmsnorm": RooflinePoint("ar_residual_rmsnorm", res["ar_rmsnorm_us"] * 1e-6,
                                        nvlink_bytes=(W - 1) * B * H * 2).report(),
    }
    out["tp_kernels"] = res
    fused.shutdown()


def _engine(kw, model=None):
    from llmctl_b200.comms import mesh
    from llmctl_b200.models.config import ModelConfig
    from llmctl_b200.runtime.engine import TrainingEngine, create_training_config
    cfg = model or ModelConfig(name="mg", layers=2, hidden=1024, ffn=2816, heads=8, vocab_size=8192, max_position_embeddings=512)
    base = dict(model_name_or_path="gpt-125m", output_dir=tempfile.mkdtemp(), batch_size=2, seq_len=256, max_steps=4,
                logging_steps=1, eval_steps=0, save_steps=0, learning_rate=1e-3, log_level="warning", metrics_jsonl=False, seed=11)
    base.update(kw)
    eng = TrainingEngine(create_training_config(**base))
    eng.config.model_name_or_path = cfg
    eng.load_model_and_tokenizer(); eng.prepare_datasets()
    return eng


def case_k7_kernels(out):
    """K7 against an fp32 PyTorch oracle, independent of the NCCL path: random per-rank gradients are written into the
    buckets, reduced + clipped + AdamW-stepped by the fused kernels, and compared with all_reduce(fp32) + the AdamW
    formula.  Covers ZeRO-1 (persistent buckets, parameter push) with NVLS and with P2P transport (the two pushes must
    agree bit for bit), ZeRO-2 (transient bucket slots) and ZeRO-3 (local shard only), two steps each."""
    import torch.nn as nn
    from llmctl_b200.comms import mesh
    from llmctl_b200.parallel.zero import ZeroOptimizer
    world, rank = dist.get_world_size(), dist.get_rank()
    res = {}
    lr, b1, b2, eps, wd, clip = 1e-2, 0.9, 0.95, 1e-8, 0.1, 1.0
    final = {}
    for tag, stage, env in (("z1_nvls", 1, {}), ("z1_p2p", 1, {"LLMCTL_K7_NVLS": "0"}), ("z2", 2, {}), ("z3", 3, {}),
                            ("z1_nvls_push_only", 1, {"LLMCTL_K7_NVLS_REDUCE": "0"})):
        mesh.reset_state()
        st = mesh.init_mesh(dp=world)
        for k in ("LLMCTL_K7_NVLS", "LLMCTL_K7_NVLS_REDUCE"):
            os.environ.pop(k, None)
        os.environ.update(env)
        torch.manual_seed(5)
        model = nn.Sequential(*[nn.Linear(512, 384 + 128 * i, bias=False) for i in range(5)]).cuda().bfloat16()
        units = [(f"l{i}", m) for i, m in enumerate(model)]
        opt = ZeroOptimizer(model, lr=lr, betas=(b1, b2), eps=eps, weight_decay=wd, zero_stage=stage, grad_clip=clip,
                            units=units, state=st, comm="native")
        assert opt.native_comm is not None, "K7 path not enabled"
        # oracle state: fp32 master of the whole (unpadded) parameter set
        with opt.full_params_context():
            ref_p = [p.detach().float().clone() for p in model.parameters()]
        ref_m = [torch.zeros_like(p) for p in ref_p]
        ref_v = [torch.zeros_like(p) for p in ref_p]
        errs = []
        gen = torch.Generator(device="cuda").manual_seed(100 + rank)
        for step in range(1, 3):
            gsum = []
            opt.set_micro_batch(0, 1)
            for u in reversed(opt.units):                      # backward order
                opt._pre_backward(u)
                for p in u.params:
                    g = torch.randn(p.shape, device="cuda", generator=gen) * (0.5 + rank)
                    p.main_grad.copy_(g)
                    gf = p.main_grad.float().clone()
                    dist.all_reduce(gf)
                    gsum.append((p, gf / world))
                for p in u.params:
                    u._param_grad_ready(p)
            gmap = {id(p): g for p, g in gsum}
            norm_ref = torch.sqrt(sum((g.double() ** 2).sum() for g in gmap.values())).float()
            gn = opt.step(lr)
            torch.cuda.synchronize()
            coef = min(1.0, clip / (float(norm_ref) + 1e-6))
            for i, p in enumerate(model.parameters()):
                g = gmap[id(p)] * coef
                ref_m[i] = b1 * ref_m[i] + (1 - b1) * g
                ref_v[i] = b2 * ref_v[i] + (1 - b2) * g * g
                mh, vh = ref_m[i] / (1 - b1 ** step), ref_v[i] / (1 - b2 ** step)
                ref_p[i] = ref_p[i] * (1 - lr * wd) - lr * mh / (vh.sqrt() + eps)
            assert abs(float(gn) - float(norm_ref)) < 1e-2 * float(norm_ref), f"{tag}: norm {float(gn)} vs {float(norm_ref)}"
            with opt.full_params_context():
                got = [p.detach().float().clone() for p in model.parameters()]
            num = sum(((a - b.bfloat16().float()) ** 2).sum() for a, b in zip(got, ref_p)).sqrt().item()
            den = sum((b ** 2).sum() for b in ref_p).sqrt().item()
            upd = lr * sum(p.numel() for p in ref_p) ** 0.5        # size of one AdamW step (|m/sqrt(v)| ~ 1)
            errs.append(num / upd)
            assert num < 0.05 * upd, f"{tag} step {step}: parameter error {num} vs update size {upd}"
        with opt.full_params_context():
            flat = torch.cat([p.detach().reshape(-1) for p in model.parameters()]).clone()
        ref = flat.clone(); dist.broadcast(ref, src=0)
        assert torch.equal(flat, ref), f"{tag}: ranks hold different parameters"
        final[tag] = flat
        res[tag] = {"err_over_update": errs, "grad_norm": float(gn)}
        torch.cuda.synchronize(); dist.barrier()
    # the NVLS push must reproduce the P2P push exactly when the reduction is the same (rank-ordered pull)
    assert torch.equal(final["z1_nvls_push_only"], final["z1_p2p"]), "multimem.st push differs from P2P push"
    for k in ("LLMCTL_K7_NVLS", "LLMCTL_K7_NVLS_REDUCE"):
        os.environ.pop(k, None)
    mesh.reset_state()
    out["k7_kernels"] = res


def _zero_traj(stage, comm, steps=4, tp=1):
    from llmctl_b200.comms import mesh
    from llmctl_b200.parallel.zero import ZeroOptimizer
    from llmctl_b200.runtime.engine import LRSchedule
    eng = _engine(dict(zero_stage=stage, tensor_parallel=tp, sequence_parallel=tp > 1))
    c = eng.config
    eng.optimizer = ZeroOptimizer(eng.model, lr=c.learning_rate, betas=tuple(c.betas), eps=c.adam_eps, weight_decay=c.weight_decay,
                                  zero_stage=stage, grad_clip=c.gradient_clipping, state=eng.state, comm=comm)
    eng.scheduler = LRSchedule(c.learning_rate, 0, 100, "constant")
    with eng.optimizer.full_params_context():
        p_init = torch.cat([p.detach().float().reshape(-1) for p in eng.model.parameters()])
    losses = []
    for _ in range(steps):
        o = eng.train_step()
        losses.append((eng._reduce_scalar(o["loss"]), float(o["grad_norm"])))
    with eng.optimizer.full_params_context():
        p_end = torch.cat([p.detach().float().reshape(-1) for p in eng.model.parameters()])
    info = {"native": eng.optimizer.native_comm is not None, "gatherer": eng.optimizer.gatherer is not None,
            "k8": dict(eng.optimizer.gatherer.stats) if eng.optimizer.gatherer is not None else None}
    torch.cuda.synchronize(); dist.barrier()
    from llmctl_b200.comms import fused
    fused.shutdown()
    mesh.reset_state()
    return losses, p_end - p_init, info


def _compare_zero(out, key, stage, tp=1):
    ref_l, ref_d, _ = _zero_traj(stage, "nccl", tp=tp)
    nat_l, nat_d, info = _zero_traj(stage, "native", tp=tp)
    assert info["native"], "K7 path was not enabled"
    if stage >= 3:
        assert info["gatherer"], "peer gatherer was not enabled"
        if tp == 1:      # every block's QKV GEMM consumed its weight through the arrival flags (K8)
            assert info["k8"]["gated_gemms"] >= 4 * 2, info
    for (la, ga), (lb, gb) in zip(ref_l, nat_l):
        assert abs(la - lb) < 1e-2 * max(1, abs(la)), f"loss nccl {ref_l} native {nat_l}"
        assert abs(ga - gb) < 2e-2 * max(1, abs(ga)), f"gnorm nccl {ref_l} native {nat_l}"
    # gate relative to the size of the update itself: a path that skipped (or halved) the update fails
    rel = ((nat_d - ref_d).norm() / ref_d.norm()).item()
    assert ref_d.norm().item() > 0 and rel < 0.1, f"update differs from the NCCL path by {rel:.3f} of its size"
    out[key] = {"nccl": ref_l, "native": nat_l, "update_rel_diff": rel, "k8": info.get("k8")}


def case_zero_native(out):
    """K7 in the engine (ZeRO-1): loss / grad-norm trajectory and the accumulated parameter update vs the NCCL path."""
    _compare_zero(out, "zero_native", 1)


def case_zero2_native(out):
    _compare_zero(out, "zero2_native", 2)


def case_zero_tp_native(out):
    """K7 on a DP x TP mesh (tp = 2 with sequence parallelism, dp = world / 2): the DP group is a sub-group, the
    gradient norm also needs the TP ranks' contributions (handed to the kernel as a device scalar)."""
    assert dist.get_world_size() >= 4 and dist.get_world_size() % 2 == 0, "needs >= 4 GPUs"
    _compare_zero(out, "zero1_tp2_native", 1, tp=2)
    _compare_zero(out, "zero3_tp2_native", 3, tp=2)


def case_zero3_native(out):
    """ZeRO-3: K7 on transient buckets + peer-memory parameter gather (+prefetch) vs NCCL collectives."""
    _compare_zero(out, "zero3_native", 3)


def case_tp_sp_engine(out):
    """TP=world + SP training with the fused K1/K2 linears (forced on, not auto-selected) vs the NCCL collectives;
    the fused arm must really have launched K1 and K2 in forward and backward."""
    from llmctl_b200.comms import fused, mesh
    res = {}
    os.environ["LLMCTL_K1"] = "fused"
    for mode in ("nccl", "fused"):
        eng = _engine(dict(tensor_parallel=dist.get_world_size(), sequence_parallel=True))
        if mode == "fused":
            assert fused.init_tp_workspace(max_tokens=2 * 256, hidden=1024) is not None
        else:
            fused.shutdown()
        eng.setup_optimizer_and_scheduler()
        res[mode] = [eng._reduce_scalar(eng.train_step()["loss"]) for _ in range(4)]
        if mode == "fused":
            rep = fused.path_report()
            res["paths"] = rep
            # per step and layer: 2 K1 + 2 K2 forward, 2 K1 + 2 K2 backward
            assert rep["calls"]["k1_fused"] >= 4 * 2 * 4 and rep["calls"]["k2_fused"] >= 4 * 2 * 4 and rep["calls"]["k1_nccl"] == 0, rep
        torch.cuda.synchronize(); dist.barrier()
        fused.shutdown(); mesh.reset_state()
    os.environ.pop("LLMCTL_K1", None)
    for a, b in zip(res["nccl"], res["fused"]):
        assert abs(a - b) < 3e-2 * max(1, abs(a)), f"{res}"
    out["tp_sp_engine"] = res


def case_vocab_ce(out):
    """K15 on the TP path: vocab-parallel cross-entropy through the native partial / finalize kernels vs fp32
    F.cross_entropy on the full logits (loss and gradient), with ignored rows."""
    import torch.nn.functional as F
    from llmctl_b200.comms import mesh
    from llmctl_b200.parallel import tp as tpl
    world, rank = dist.get_world_size(), dist.get_rank()
    mesh.reset_state()
    mesh.init_mesh(tp=world)
    torch.manual_seed(77)
    rows, V = 1000, 4096 * world
    full = (3.0 * torch.randn(rows, V, device="cuda")).bfloat16()
    targets = torch.randint(0, V, (rows,), device="cuda")
    targets[::7] = -100
    ref_in = full.float().requires_grad_(True)
    ref = F.cross_entropy(ref_in, targets, ignore_index=-100) * 0.5
    ref.backward()
    vl = V // world
    shard = full[:, rank * vl:(rank + 1) * vl].contiguous().requires_grad_(True)
    logits = shard * 1.0                       # non-leaf, as produced by the LM-head GEMM
    from llmctl_b200.ops import native
    before = native.launch_count
    loss = tpl.vocab_parallel_cross_entropy(logits, targets, grad_scale=0.5)
    assert native.launch_count - before == 2, "native partial/finalize kernels were not used"
    loss.backward()
    gref = ref_in.grad[:, rank * vl:(rank + 1) * vl]
    e_loss = abs(float(loss) - float(ref)) / abs(float(ref))
    e_grad = (shard.grad.float() - gref).abs().max().item() / gref.abs().max().item()
    assert e_loss < 1e-3 and e_grad < 2e-2, (e_loss, e_grad)
    assert shard.grad[::7].abs().max().item() == 0.0, "ignored rows must get zero gradient"
    mesh.reset_state()
    out["vocab_ce"] = {"loss_rel_err": e_loss, "grad_rel_err": e_grad}


def case_watchdog(out):
    """A rank that never launches its side of a collective: the waiting kernel must give up after the deadline,
    report what it was waiting for, and the communicator must be usable again afterwards."""
    import time
    from llmctl_b200.comms import symm
    from llmctl_b200.comms.collectives import PeerCollectives
    rank, world = dist.get_rank(), dist.get_world_size()
    pc = PeerCollectives(1 << 16)
    n = 4096
    pc.buf.tensor[:n].fill_(float(rank + 1))
    torch.cuda.synchronize(); dist.barrier()
    ref = pc.all_reduce(n, algo="oneshot").float().clone()
    torch.cuda.synchronize()
    assert symm.watchdog_poll() is None
    symm.set_watchdog_timeout_ms(300)
    dist.barrier()
    t0 = time.perf_counter()
    if rank == 0:
        pc.all_reduce(n, algo="oneshot")          # peers skip this epoch on purpose
    else:
        pc.epoch += 1
    torch.cuda.synchronize()
    waited = time.perf_counter() - t0
    rec = symm.watchdog_poll()
    if rank == 0:
        assert rec is not None and rec["timed_out_waits"] >= 1 and rec["module"] == "collectives", rec
        assert 0.25 < waited < 5.0, waited
    else:
        assert rec is None, rec
    symm.set_watchdog_timeout_ms(30000)
    dist.barrier()
    # randomised launch skew: every rank delays its launch by a different amount each round
    g = torch.Generator().manual_seed(1234 + rank)
    for it in range(12):
        pc.buf.tensor[:n].fill_(float(rank + 1))
        torch.cuda.synchronize(); dist.barrier()
        torch.cuda._sleep(int(torch.randint(0, 3_000_000, (1,), generator=g)))
        got = pc.all_reduce(n, algo="oneshot").float()
        assert torch.equal(got, ref), f"round {it}: all-reduce under launch skew differs"
        torch.cuda.synchronize()
    assert symm.watchdog_poll() is None
    out["watchdog"] = {"first_record": rec, "waited_s": waited, "skew_rounds": 12}


def case_tp_serving(out):
    """Tensor-parallel decode: K11 (fused all-reduce + residual + RMSNorm) vs NCCL all-reduce + ATen, same engine."""
    import time
    from llmctl_b200.comms import mesh
    from llmctl_b200.models.config import ModelConfig
    from llmctl_b200.serve import engine as E
    world = dist.get_world_size()
    mesh.reset_state()
    mesh.init_mesh(tp=world)
    torch.manual_seed(1234 + dist.get_rank())
    cfg = ModelConfig(name="serve-tp", layers=4, hidden=1024, ffn=2816, heads=8, vocab_size=4096, max_position_embeddings=1024)
    orig = E.resolve_model
    E.resolve_model = lambda spec: cfg
    try:
        eng = E.InferenceEngine("serve-tp", max_batch_size=8, max_batch_tokens=8192, num_kv_blocks=512)
    finally:
        E.resolve_model = orig
    assert eng._ar is not None, "fused TP decode context was not created"
    g = torch.Generator().manual_seed(7)
    prompts = [torch.randint(3, 4000, (n,), generator=g).tolist() for n in (33, 64, 17, 128, 50, 77, 90, 12)]
    res = {}
    ar = eng._ar
    toks = {}
    for mode in ("fused", "nccl", "fused"):
        eng._ar = ar if mode == "fused" else None
        torch.cuda.synchronize(); dist.barrier()
        t0 = time.perf_counter()
        toks[mode] = eng.generate(prompts, max_tokens=24, temperature=0.0)
        torch.cuda.synchronize()
        res[mode + "_s"] = time.perf_counter() - t0
        res[mode + "_decode_step_ms"] = 1e3 * eng.stats["decode_time_s"] / max(eng.stats["decode_steps"], 1)
        eng.stats["decode_time_s"], eng.stats["decode_steps"] = 0.0, 0
    agree = sum(int(a == b) for x, y in zip(toks["fused"], toks["nccl"]) for a, b in zip(x, y))
    total = sum(len(x) for x in toks["fused"])
    first = sum(int(x[0] == y[0]) for x, y in zip(toks["fused"], toks["nccl"]))
    second = sum(int(x[1] == y[1]) for x, y in zip(toks["fused"], toks["nccl"]))     # first token out of the decode path
    res.update(agree=agree, total=total, first_token_agree=first, second_token_agree=second)
    # all TP ranks must have produced the same tokens
    mine = torch.tensor([t for x in toks["fused"] for t in x], device="cuda")
    ref = mine.clone(); dist.broadcast(ref, src=0)
    assert torch.equal(mine, ref), "TP ranks diverged"
    # a random-init model has nearly flat logits: one bf16-rounding flip changes the rest of that sequence, so only
    # the tokens before the first possible flip are required to match everywhere
    assert first == len(prompts) and second >= len(prompts) - 1 and agree >= 0.5 * total, res
    from llmctl_b200.comms import symm
    assert symm.watchdog_poll() is None
    out["tp_serving"] = res


CASES = {"vocab_ce": case_vocab_ce, "tp_serving": case_tp_serving, "watchdog": case_watchdog, "probe": case_probe, "tp_kernels": case_tp_kernels, "k7_kernels": case_k7_kernels, "zero_native": case_zero_native, "zero2_native": case_zero2_native, "zero_tp_native": case_zero_tp_native,
         "zero3_native": case_zero3_native,
         "tp_sp_engine": case_tp_sp_engine}


def main():
    names = sys.argv[1:] or list(CASES)
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    out = {}
    failed = []
    for n in names:
        try:
            CASES[n](out)
        except Exception as e:  # noqa: BLE001
            import traceback
            failed.append(n)
            out[n + "_error"] = f"{type(e).__name__}: {e}"
            if dist.get_rank() == 0:
                traceback.print_exc()
            break     # ranks may now be out of step: stop here
    if dist.get_rank() == 0:
        print("MGPU_RESULT " + json.dumps(out, default=str))
    dist.destroy_process_group()
    sys.exit(1 if failed else 0)


if __name__ == "__main__":
    main()
