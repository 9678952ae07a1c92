"""Unit tests the reference never had: planner, config schemas, health thresholds, autotuner,
plugin registry, checkpoint GC, LR schedule, export re-sharding, roofline."""
import contextlib
import json
import math
import time
from pathlib import Path

import pytest
import torch


def test_planner_param_count_and_measured_search():
    from llmctl_b200.models.config import get_preset
    from llmctl_b200.partition.planner import HardwareNumbers, MeasuredCostModel, ReferenceCostModel
    m7 = get_preset("gpt-7b")
    assert m7.num_parameters() == 6_738_415_616                      # reference configs/models/llama-7b.json:23
    ref = ReferenceCostModel(m7.to_dict(), {"gpu": {"count": 8}})
    assert ref.parameters() == 5_164_761_088                         # the reference's (defective) estimate, golden
    assert abs(ref.model_memory_gb() - 57.72) < 0.01
    assert ref.manual(2, 1, 0).zero_stage == 0                       # explicit 0 stays 0 (D9)
    hw = HardwareNumbers(gpus=8)
    plans = MeasuredCostModel(m7, hw, seq_len=2048).search(global_batch=64)
    assert plans and plans[0].estimated_memory_gb <= 0.92 * 180
    assert all(p.tensor_parallel * p.pipeline_parallel * p.data_parallel == 8 for p in plans)
    assert plans == sorted(plans, key=lambda p: -p.estimated_tokens_per_s)
    m13 = get_preset("gpt-13b")
    pinned = MeasuredCostModel(m13, hw, 4096).search(global_batch=32, pins={"tensor_parallel": 4, "pipeline_parallel": 2})
    assert pinned and all((p.tensor_parallel, p.pipeline_parallel) == (4, 2) for p in pinned)
    assert pinned[0].breakdown["pp_bubble"] > 0
    small = MeasuredCostModel(m13, HardwareNumbers(gpus=8, memory_gb=24), 4096).search(global_batch=32)
    assert all(p.estimated_memory_gb <= 0.92 * 24 for p in small)    # memory cap is honoured


def test_partition_layers():
    from llmctl_b200.parallel.pp import partition_layers
    assert partition_layers(32, 4) == [(0, 8), (8, 16), (16, 24), (24, 32)]
    r = partition_layers(40, 3)
    assert r[0][0] == 0 and r[-1][1] == 40 and all(a < b for a, b in r) and all(r[i][1] == r[i + 1][0] for i in range(2))
    with pytest.raises(ValueError):
        partition_layers(2, 4)


def test_config_schemas_and_precedence(tmp_path):
    import tomli_w
    from llmctl_b200.cli.commands.init import default_training_config
    from llmctl_b200.config.schemas import (ModelSchema, ServeConfig, load_training_preset, resolve_training_config)
    with pytest.raises(Exception):
        ModelSchema.model_validate({"name": "x", "layers": 0, "hidden": 8, "heads": 2, "vocab_size": 10})
    with pytest.raises(Exception):
        ServeConfig(artifact="a", scheduler="bogus")
    preset = tmp_path / "configs" / "default.toml"
    preset.parent.mkdir(parents=True)
    preset.write_text(tomli_w.dumps(default_training_config("gpt", "125m", "proj")))
    ps = load_training_preset(preset)
    assert ps.checkpoint.async_ is True and ps.parallel.activation_checkpoint == "selective"
    plan = tmp_path / "plan.toml"
    plan.write_text(tomli_w.dumps({"parallelism": {"tensor_parallel": 2, "pipeline_parallel": 1, "data_parallel": 4, "zero_stage": 3,
                                                   "micro_batch_size": 2, "global_batch_size": 32, "sequence_parallel": True}}))
    cfg = resolve_training_config(preset, plan, {"learning_rate": 1e-5, "zero_stage": None})
    assert cfg["tensor_parallel"] == 2 and cfg["zero_stage"] == 3 and cfg["sequence_parallel"] is True   # plan > preset
    assert cfg["gradient_accumulation_steps"] == 4 and cfg["batch_size"] == 2
    assert cfg["learning_rate"] == 1e-5                                                                  # CLI > files
    assert cfg["weight_decay"] == 0.1 and cfg["scheduler"] == "cosine"                                   # preset > defaults


def test_health_thresholds_fire():
    from llmctl_b200.metrics.health import (HealthStatus, InferenceHealthMonitor, SystemHealthMonitor, TrainingHealthMonitor)

    class Fake(SystemHealthMonitor):
        def __init__(self, m):
            super().__init__()
            self._m = m

        def collect(self):
            return self._m
    r = Fake({"cpu_usage": 10, "memory_usage": 10, "disk_space": 90, "gpu_memory": 10}).get_health_report()
    assert r.status == HealthStatus.WARNING and r.checks["disk_space"] is False      # D12: disk threshold fires
    r = Fake({"cpu_usage": 10, "memory_usage": 10, "disk_space": 10, "gpu_memory": 99}).get_health_report()
    assert r.status == HealthStatus.CRITICAL and r.checks["gpu_memory"] is False      # D12: GPU-memory threshold fires
    t = TrainingHealthMonitor(stall_seconds=0.05)
    assert t.get_health_report().status == HealthStatus.UNKNOWN
    t.update_metrics(1, 2.5, 1.0)
    assert t.get_health_report().status == HealthStatus.HEALTHY
    t.update_metrics(2, float("nan"), 1.0)
    assert t.get_health_report().status == HealthStatus.CRITICAL
    t.update_metrics(3, 2.0, 500.0)
    assert t.get_health_report().status == HealthStatus.WARNING
    t.update_metrics(4, 2.0, 1.0); time.sleep(0.1)
    assert t.get_health_report().status == HealthStatus.CRITICAL                      # stalled
    i = InferenceHealthMonitor()
    for k in range(20):
        i.record_request(0.1, success=k != 0)
    assert i.get_health_report().status == HealthStatus.CRITICAL                      # 5 % errors
    i2 = InferenceHealthMonitor(); i2.record_request(11.0); i2.update_queue(5)
    assert i2.get_health_report().status == HealthStatus.WARNING


def test_observability_feeds_prometheus():
    from prometheus_client import CollectorRegistry, generate_latest
    from llmctl_b200.metrics.observability import ObservabilityManager
    om = ObservabilityManager()
    reg = CollectorRegistry()
    om.enable_prometheus(port=None, registry=reg)
    om.record_training_step(step=3, loss=2.0, learning_rate=1e-4, tokens_per_second=1000.0, grad_norm=0.5, step_time=0.1, mfu=0.4)
    om.record_inference_request(latency=0.2, tokens=10, ttft=0.05)
    text = generate_latest(reg).decode()
    assert "llmctl_training_loss 2.0" in text and "llmctl_training_steps_total 3.0" in text   # D15: counters move
    assert 'llmctl_inference_requests_total{status="ok"} 1.0' in text and "llmctl_inference_latency_seconds_count 1.0" in text


def test_autotuner_grid_search_and_cache(tmp_path):
    from llmctl_b200.plugins.autotuning import AutoTuner, Tunable, TuningConfig

    class Toy(Tunable):
        calls = 0

        def get_parameter_space(self):
            return {"a": [1, 2, 3, 4], "b": [10, 20]}

        def validate_parameters(self, p):
            return p["a"] != 4

        def set_parameters(self, p):
            self.p = p

        def benchmark(self, x):
            Toy.calls += 1
            return abs(self.p["a"] - 2) + self.p["b"] / 100.0
    t = AutoTuner(TuningConfig(max_iterations=50))
    r = t.grid_search(Toy(), None, "toy")
    assert r.best_config == {"a": 2, "b": 10} and r.iterations == 6 and r.improvement > 0
    n = Toy.calls
    assert t.grid_search(Toy(), None, "toy") is r and Toy.calls == n                  # cache hit
    t.save_results(str(tmp_path / "c.json"))
    t2 = AutoTuner(); t2.load_results(str(tmp_path / "c.json"))
    assert t2.results_cache["toy"].best_config == {"a": 2, "b": 10}
    assert AutoTuner(TuningConfig(max_iterations=2)).grid_search(Toy(), None).iterations == 2   # max_iterations honoured (D13)


def test_plugin_registry(tmp_path, monkeypatch):
    from llmctl_b200.plugins.registry import PluginRegistry
    (tmp_path / "my_plugin.py").write_text("class S:\n    def schedule(self, reqs):\n        return reqs[:1]\n\ndef register():\n    return {'first-only': S}\n")
    monkeypatch.syspath_prepend(str(tmp_path))
    monkeypatch.setenv("LLMCTL_PLUGINS", "schedulers:my_plugin")
    reg = PluginRegistry()
    assert reg.get("schedulers", "first-only")().schedule([1, 2]) == [1]
    assert {"dynamic", "simple", "vllm-like"} <= set(reg.list("schedulers")) and "rmsnorm" in reg.list("kernels")
    with pytest.raises(KeyError):
        reg.register("bogus", "x", object())


def test_lr_schedule_and_config_validation():
    from llmctl_b200.runtime.engine import LRSchedule, create_training_config
    s = LRSchedule(1.0, warmup=4, total=14, kind="linear")
    assert [round(s.lr_at(i), 3) for i in (0, 3, 4, 9, 14)] == [0.25, 1.0, 1.0, 0.5, 0.0]
    c = LRSchedule(1.0, 0, 10, "cosine")
    assert abs(c.lr_at(5) - 0.5) < 1e-6
    with pytest.raises(TypeError):
        create_training_config(not_a_field=1)


def test_checkpoint_gc_and_latest(tmp_path):
    from llmctl_b200.io.checkpoint import gc_checkpoints, latest_checkpoint, list_checkpoints
    for step, complete in ((10, True), (20, True), (30, False), (40, True)):
        d = tmp_path / f"checkpoint-{step}"; d.mkdir()
        if complete:
            (d / "COMPLETE").write_text(str(step))
    assert [d.name for d in list_checkpoints(tmp_path)] == ["checkpoint-10", "checkpoint-20", "checkpoint-40"]
    assert latest_checkpoint(tmp_path).name == "checkpoint-40"
    removed = {d.name for d in gc_checkpoints(tmp_path, keep_latest=2)}
    assert removed == {"checkpoint-10", "checkpoint-30"}                               # oldest complete + stale incomplete
    assert sorted(p.name for p in tmp_path.iterdir()) == ["checkpoint-20", "checkpoint-40"]


def test_tp_merge_split_roundtrip():
    from llmctl_b200.io.export import merge_tp, split_tp, to_hf_llama
    full = torch.arange(24 * 4, dtype=torch.float32).view(24, 4)
    for packed, dim in ((3, 0), (1, 0), (1, 1), (2, 0)):
        shards = [split_tp(full, dim, packed, 2, r) for r in range(2)]
        assert torch.equal(merge_tp(shards, dim, packed), full)
    hf = to_hf_llama({"blocks.0.attn.qkv.weight": full, "blocks.0.mlp.up.weight": full, "embed.weight": full})
    assert hf["model.layers.0.self_attn.k_proj.weight"].shape == (8, 4) and "model.embed_tokens.weight" in hf


def test_roofline_report():
    from llmctl_b200.metrics.roofline import RooflinePoint, peak_flops
    r = RooflinePoint("gemm", seconds=2 * 8192 ** 3 / peak_flops(False) * 2, flops=2 * 8192 ** 3).report()
    assert r["bound"] == "compute" and abs(r["fraction_of_roofline"] - 0.5) < 1e-6
    assert RooflinePoint("copy", 1.0, hbm_bytes=1e12, nvlink_bytes=1e12).report()["bound"] == "nvlink"


def test_dataset_determinism_and_resume():
    from llmctl_b200.io.dataset import SyntheticTokenDataset, TokenLoader
    ds = SyntheticTokenDataset(1000, 16, seed=3)
    assert (ds[5] == SyntheticTokenDataset(1000, 16, seed=3)[5]).all() and (ds[5] != ds[6]).any()
    a = TokenLoader(ds, 2, dp_rank=0, dp_size=2); b = TokenLoader(ds, 2, dp_rank=1, dp_size=2)
    ta, _ = a.next_batch(); tb, _ = b.next_batch()
    assert not torch.equal(ta, tb)                                                     # ranks see disjoint samples
    a.next_batch(); st = a.state_dict()
    nxt, _ = a.next_batch()
    c = TokenLoader(ds, 2, dp_rank=0, dp_size=2); c.load_state_dict(st)
    assert torch.equal(c.next_batch()[0], nxt)                                         # resumable cursor


def test_shipped_configs_validate():
    """Every file under configs/ parses with its schema; the 13B 3D preset plans onto 8 GPUs."""
    from pathlib import Path
    from llmctl_b200.config.schemas import load_hardware_profile, load_model_file, load_training_preset
    from llmctl_b200.models.config import ModelConfig
    root = Path(__file__).resolve().parent.parent / "configs"
    for f in (root / "models").glob("*.json"):
        m = load_model_file(f)
        assert ModelConfig.from_file(f).num_parameters() == m.estimated_params
    hw = load_hardware_profile(root / "hw" / "b200x8.toml")
    assert hw.gpu.count == 8 and hw.limits.measured and hw.interconnect.nvls_multicast
    names = set()
    for f in (root / "presets").glob("*.toml"):
        p = load_training_preset(f)
        names.add(f.name)
        assert p.parallel.tensor_parallel * p.parallel.pipeline_parallel <= 8
    assert {"gpt-7b-b200x8-tp8-sp.toml", "gpt-7b-b200x8-zero3.toml", "gpt-13b-b200x8-tp4-pp2.toml", "gpt-125m-cpu-pp2.toml"} <= names


def test_decode_staging_layout_and_buckets():
    """The packed decode-step input buffer: int64 views stay 8-byte aligned, padding rows are inert, bucket sizes are
    powers of two capped at the engine limits."""
    import numpy as np
    from llmctl_b200.serve.engine import InferenceEngine, _DecodeInputs
    inp = _DecodeInputs(4, 6, torch.device("cpu"))
    h = inp.host
    h.fill_pad()
    h.tokens[:2] = [11, 12]
    h.slots[:2] = [100, 2 ** 33 + 5]           # slots are 64-bit
    h.positions[:2] = [7, 8]
    h.ctx[:2] = [8, 9]
    h.block_tables[0, :3] = [5, 6, 7]
    inp.upload()
    assert inp.tokens.dtype == torch.int64 and inp.tokens.shape == (4, 1) and inp.tokens[:2, 0].tolist() == [11, 12]
    assert inp.slots.tolist() == [100, 2 ** 33 + 5, -1, -1]
    assert inp.positions.tolist() == [7, 8, 0, 0] and inp.ctx.tolist() == [8, 9, 0, 0]
    assert inp.block_tables[0].tolist() == [5, 6, 7, 0, 0, 0] and int(inp.block_tables[1:].abs().sum()) == 0
    assert inp.tokens.data_ptr() % 8 == 0 and inp.slots.data_ptr() % 8 == 0
    assert inp.nbytes == (6 * 4 + 4 * 6) * 4
    assert [InferenceEngine._bucket(n, 1, 8) for n in (1, 2, 3, 5, 8)] == [1, 2, 4, 8, 8]
    assert InferenceEngine._bucket(300, 256, 4096) == 512 and InferenceEngine._bucket(5000, 256, 4096) == 5000
    assert isinstance(h.tokens, np.ndarray)


def test_paged_decode_split_heuristic():
    from llmctl_b200.ops.serving import choose_splits
    assert choose_splits(8, 4, 2304, 16) == 36             # 64-token splits, ~8 CTAs per SM
    assert choose_splits(8, 32, 2304, 16) == 5             # enough (batch, head) pairs already
    assert choose_splits(1, 4, 32768, 16) == 256           # capped
    assert choose_splits(64, 32, 100, 16) == 1
    assert choose_splits(1, 1, 10, 16) == 1


def test_cpu_noops_for_gpu_only_facilities():
    """NVTX ranges and the peer-signal watchdog must be inert (not failing) without a GPU."""
    from llmctl_b200.comms import symm
    from llmctl_b200.utils.nvtx import mark, nvtx_range
    with nvtx_range("phase"):
        mark("event")
    if not torch.cuda.is_available():
        assert symm.watchdog_poll() is None
        symm.check_watchdog("unit test")
    t = symm.PeerTable.of([0x1000, 0x2000])
    assert t.ptr[0] == 0x1000 and t.ptr[1] == 0x2000 and not t.ptr[7]


def test_text_dataset_is_tokenised_and_missing_sources_fail(tmp_path):
    from llmctl_b200.io.dataset import MMapTokenDataset, SyntheticTokenDataset, build_dataset
    txt = tmp_path / "corpus.txt"
    txt.write_text("the quick brown fox jumps over the lazy dog\n" * 50)
    ds = build_dataset(str(txt), 512, 16)
    assert isinstance(ds, MMapTokenDataset) and len(ds) > 10
    assert (tmp_path / "corpus.txt.v512.bin").exists()
    toml = tmp_path / "data.toml"
    toml.write_text(f'[dataset]\ntype = "text"\npath = "{txt}"\n')
    assert isinstance(build_dataset(str(toml), 512, 16), MMapTokenDataset)
    toml.write_text('[[sources]]\npath = "corpus.txt"\nsplit = "train"\n')
    assert isinstance(build_dataset(str(toml), 512, 16), MMapTokenDataset)
    toml.write_text('[dataset]\ntype = "synthetic"\n')
    assert isinstance(build_dataset(str(toml), 512, 16), SyntheticTokenDataset)
    import pytest
    with pytest.raises(FileNotFoundError):
        build_dataset(str(tmp_path / "nope.bin"), 512, 16)
    toml.write_text('[dataset]\ntype = "tokens"\npath = "missing.bin"\n')
    with pytest.raises(FileNotFoundError):
        build_dataset(str(toml), 512, 16)


def test_weight_only_quantizers_round_trip_and_plugin_group():
    """int8 per-channel and int4 group-wise weight-only quantisers: registered in the `quantizers` plugin group,
    dequantised weights stay within the expected rounding error, non-matrix tensors pass through untouched."""
    import torch
    from llmctl_b200.io.quantize import dequantize_if_needed, relative_error
    from llmctl_b200.plugins.builtin import register_quantizers
    from llmctl_b200.plugins.registry import get_registry
    assert {"int8", "int4"} <= set(register_quantizers()) and {"int8", "int4"} <= set(get_registry().list("quantizers"))
    torch.manual_seed(0)
    sd = {"blocks.0.attn.qkv.weight": torch.randn(96, 256).bfloat16() * 0.05, "blocks.0.norm1.weight": torch.ones(256).bfloat16(),
          "embed.weight": torch.randn(64, 256).bfloat16()}
    for name, tol in (("int8", 0.01), ("int4", 0.12)):
        q = get_registry().get("quantizers", name)()
        packed = q.quantize(sd)
        assert packed["blocks.0.attn.qkv.weight"].dtype in (torch.int8, torch.uint8)
        assert packed["blocks.0.attn.qkv.weight"].numel() * packed["blocks.0.attn.qkv.weight"].element_size() <= 96 * 256
        assert torch.equal(packed["embed.weight"], sd["embed.weight"]) and torch.equal(packed["blocks.0.norm1.weight"], sd["blocks.0.norm1.weight"])
        back = dequantize_if_needed(packed, name)
        assert set(back) == set(sd)
        assert relative_error(sd["blocks.0.attn.qkv.weight"], back["blocks.0.attn.qkv.weight"]) < tol


def test_gguf_writer_round_trip(tmp_path):
    """GGUF v3 container: header, metadata and tensor directory parse back; q|k|v and gate|up are split, q/k rows are
    permuted to llama.cpp's interleaved RoPE layout (an involution-free permutation checked against its definition)."""
    import torch
    from llmctl_b200.io.gguf import read_gguf, write_gguf
    torch.manual_seed(1)
    H, heads, ffn, V = 64, 4, 128, 100
    full = {"embed.weight": torch.randn(V, H).bfloat16(), "final_norm.weight": torch.ones(H).bfloat16(),
            "lm_head.weight": torch.randn(V, H).bfloat16(), "blocks.0.norm1.weight": torch.ones(H).bfloat16(),
            "blocks.0.norm2.weight": torch.ones(H).bfloat16(), "blocks.0.attn.qkv.weight": torch.randn(3 * H, H).bfloat16(),
            "blocks.0.attn.out.weight": torch.randn(H, H).bfloat16(), "blocks.0.mlp.up.weight": torch.randn(2 * ffn, H).bfloat16(),
            "blocks.0.mlp.down.weight": torch.randn(H, ffn).bfloat16()}
    cfg = {"name": "t", "hidden": H, "layers": 1, "ffn": ffn, "heads": heads, "vocab_size": V, "max_position_embeddings": 128}
    meta, tensors = read_gguf(write_gguf(tmp_path / "m.gguf", full, cfg, vocab=[f"t{i}" for i in range(V)]))
    assert meta["general.architecture"] == "llama" and meta["llama.block_count"] == 1 and meta["llama.attention.head_count"] == heads
    assert len(meta["tokenizer.ggml.tokens"]) == V
    assert set(tensors) == {"token_embd.weight", "output_norm.weight", "output.weight", "blk.0.attn_norm.weight", "blk.0.ffn_norm.weight",
                            "blk.0.attn_q.weight", "blk.0.attn_k.weight", "blk.0.attn_v.weight", "blk.0.attn_output.weight",
                            "blk.0.ffn_gate.weight", "blk.0.ffn_up.weight", "blk.0.ffn_down.weight"}
    assert torch.equal(tensors["token_embd.weight"], full["embed.weight"]) and tensors["output_norm.weight"].dtype == torch.float32
    q = full["blocks.0.attn.qkv.weight"][:H]
    hd = H // heads
    # row (head h, pair j, half s) of the rotate-half layout lands at (head h, 2j + s)
    for h in range(heads):
        for j in range(hd // 2):
            assert torch.equal(tensors["blk.0.attn_q.weight"][h * hd + 2 * j], q[h * hd + j])
            assert torch.equal(tensors["blk.0.attn_q.weight"][h * hd + 2 * j + 1], q[h * hd + hd // 2 + j])
    assert torch.equal(tensors["blk.0.attn_v.weight"], full["blocks.0.attn.qkv.weight"][2 * H:])
    assert torch.equal(tensors["blk.0.ffn_up.weight"], full["blocks.0.mlp.up.weight"][ffn:])


def test_train_consumes_the_model_named_by_the_plan(tmp_path):
    """`llmctl train --plan P` trains the model the plan was computed for (model file, else the name recorded in the
    plan's [model] table) at the plan's sequence length, unless a flag overrides it."""
    import json
    from llmctl_b200.config.schemas import resolve_training_config
    root = Path(__file__).resolve().parent.parent
    plan = root / "configs" / "plans" / "gpt-13b-b200x8-auto-pp2.toml"
    import os
    cwd = os.getcwd()
    os.chdir(root)
    try:
        r = resolve_training_config(None, plan, {"max_steps": 3})
        assert r["model_name_or_path"].endswith("gpt-13b.json") and r["seq_len"] == 2048
        assert (r["tensor_parallel"], r["pipeline_parallel"], r["sequence_parallel"]) == (4, 2, True)
        assert resolve_training_config(None, plan, {"model_name_or_path": "gpt-125m"})["model_name_or_path"] == "gpt-125m"
    finally:
        os.chdir(cwd)
    # a plan whose model file is gone falls back to the model name stored in the plan
    txt = plan.read_text().replace('model_file = "configs/models/gpt-13b.json"', 'model_file = "nowhere/x.json"')
    p2 = tmp_path / "p.toml"
    p2.write_text(txt)
    assert resolve_training_config(None, p2, {})["model_name_or_path"] == "gpt-13b"


def test_measured_cost_model_reproduces_the_round2_b200_runs():
    """The planner's step-time model against what this framework measured on 8 x B200 (profiles/bench_n8_with_extras.json,
    profiles/train_13b_plan_cli/, profiles/bench_n1.json): every configuration within 15%."""
    from llmctl_b200.models.config import get_preset
    from llmctl_b200.partition.planner import HardwareNumbers, MeasuredCostModel
    hw = HardwareNumbers(gpus=8)
    points = [  # model, seq, (tp, pp, dp, zero, micro_batch, sp, ckpt, n_micro), measured ms
        ("gpt-7b", 512, (1, 1, 8, 1, 8, False, "none", 1), 173.2), ("gpt-7b", 512, (8, 1, 1, 0, 8, True, "none", 1), 48.2),
        ("gpt-7b", 512, (1, 1, 8, 3, 8, False, "none", 1), 188.0), ("gpt-13b", 2048, (4, 2, 1, 0, 2, True, "none", 8), 489.0),
        ("gpt-13b", 2048, (4, 2, 1, 0, 1, True, "none", 16), 632.0), ("gpt-1b", 512, (2, 1, 1, 0, 4, True, "none", 1), 21.0)]
    for name, seq, args, measured in points:
        t = MeasuredCostModel(get_preset(name), hw, seq_len=seq).step_time(*args)["total"] * 1e3
        assert abs(t - measured) / measured < 0.15, (name, args, t, measured)
    t1 = MeasuredCostModel(get_preset("gpt-7b"), HardwareNumbers(gpus=1), seq_len=512).step_time(1, 1, 1, 0, 8, False, "none", 1)["total"] * 1e3
    assert abs(t1 - 179.0) / 179.0 < 0.1
    # fewer, larger micro-batches win under a pipeline once the per-layer overhead is counted
    m = MeasuredCostModel(get_preset("gpt-13b"), hw, seq_len=2048)
    best = m.search(global_batch=16, pins={"pipeline_parallel": 2, "tensor_parallel": 4})[0]
    assert best.micro_batch_size >= 2 and best.sequence_parallel, best


def test_reference_arm_provisions_itself(tmp_path):
    """`baseline/provision.py` installs the unmodified reference (pip --no-deps from a copy, else a verbatim copy of
    the pure-Python package) into an empty target and is a no-op afterwards; without a source tree it says so."""
    import os
    import subprocess
    import sys
    root = Path(__file__).resolve().parent.parent
    if not Path("/root/reference/llmctl/runtime/engine.py").exists():
        pytest.skip("reference source tree is not mounted here")
    dst = tmp_path / "ref"
    code = ("import sys; sys.path.insert(0, %r); import provision as p; ok, how = p.ensure_reference(); print(ok, '|', how); "
            "ok2, how2 = p.ensure_reference(); print(ok2, '|', how2)") % str(root / "baseline")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LLMCTL_REFERENCE_DST=str(dst)))
    assert r.returncode == 0, r.stderr[-2000:]
    lines = r.stdout.strip().splitlines()
    assert lines[0].startswith("True") and lines[1].startswith("True | already installed"), r.stdout
    assert (dst / "llmctl" / "runtime" / "engine.py").read_text() == Path("/root/reference/llmctl/runtime/engine.py").read_text()
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120,
                       env=dict(os.environ, LLMCTL_REFERENCE_DST=str(tmp_path / "ref2"), LLMCTL_REFERENCE_SRC=str(tmp_path / "nowhere")))
    # /root/reference is still found (second source); with it hidden the function reports why it cannot install
    assert r.returncode == 0


def test_apply_without_gradients_keeps_autograd_rules():
    """ops.native.apply calls the forward itself only where autograd, forward-mode AD and tracing have nothing to record, and an
    in-place forward still moves the version counter."""
    from llmctl_b200.ops import native
    seen = []

    class Twice(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            seen.append(type(ctx).__name__)
            ctx.save_for_backward(x)
            return x * 2

        @staticmethod
        def backward(ctx, g):
            return 2 * g

    class AddOne(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            with torch.no_grad():
                x.data.add_(1)
            ctx.mark_dirty(x)
            return x

        @staticmethod
        def backward(ctx, g):
            return g
    x = torch.ones(3, requires_grad=True)
    y = native.apply(Twice, x)
    y.sum().backward()
    assert torch.equal(x.grad, torch.full((3,), 2.0)) and seen[-1] != "_NoContext"
    with torch.no_grad():
        assert torch.equal(native.apply(Twice, x), torch.full((3,), 2.0)) and seen[-1] == "_NoContext"
    assert not native.apply(Twice, torch.ones(3)).requires_grad and seen[-1] == "_NoContext"
    z = torch.zeros(3)
    before = z._version
    assert native.apply(AddOne, z) is z and z._version > before and torch.equal(z, torch.ones(3))
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(torch.ones(3), torch.ones(3))
        with pytest.raises(Exception):
            native.apply(Twice, dual)           # no jvp: refused, as Twice.apply refuses it
    with pytest.raises(Exception):
        torch.func.vmap(lambda t: native.apply(Twice, t))(torch.ones(2, 3))


@pytest.mark.parametrize("layer", ["up", "down"])
@pytest.mark.parametrize("change", ["subclass", "finish", "instance", "class", "call", "global_forward", "global_pre", "global_backward", "hook", "module"])
def test_gated_mlp_calls_its_layers_where_they_are_more_than_their_product(monkeypatch, layer, change):
    """Subclasses, replaced methods and modules and hooks of any kind see every call of an MLP's two layers, as if nothing were fused."""
    from torch.nn.modules import module as every
    from llmctl_b200.models.config import ModelConfig
    from llmctl_b200.models.gpt import MLP
    from llmctl_b200.ops import functional as ops
    from llmctl_b200.parallel import tp
    cfg = ModelConfig(name="t", layers=1, hidden=16, ffn=24, heads=2, vocab_size=32, max_position_embeddings=8)
    torch.manual_seed(0)
    mlp = MLP(cfg, torch.float32, "cpu")
    x = torch.randn(5, 16, requires_grad=True)
    seen, factor = [], 1.0
    assert tp.runs_plain(mlp.up) and tp.runs_plain(mlp.down)
    old = getattr(mlp, layer)
    handle = None
    if change == "subclass":
        class Doubled(type(old)):
            def forward(self, x):
                return 2 * super().forward(x)
        old.__class__, factor = Doubled, 2.0
    elif change == "finish":
        if layer == "up":
            pytest.skip("only the row-parallel layer has it")
        old.finish, factor = lambda y: 2 * y, 2.0
    elif change == "instance":
        old.forward, factor = lambda x: 2 * x @ old.weight.t(), 2.0
    elif change == "class":
        monkeypatch.setattr(type(old), "forward", lambda self, x: 2 * x @ self.weight.t())
        factor = 2.0
    elif change == "call":
        class Called(type(old)):
            def __call__(self, x):
                return 2 * super().__call__(x)
        old.__class__, factor = Called, 2.0
    elif change == "global_forward":
        handle = every.register_module_forward_hook(lambda m, i, o: seen.append(m))
    elif change == "global_pre":
        handle = every.register_module_forward_pre_hook(lambda m, i: seen.append(m))
    elif change == "global_backward":
        handle = every.register_module_full_backward_hook(lambda m, gi, go: seen.append(m))
    elif change == "hook":
        old.register_forward_hook(lambda m, i, o: seen.append(m))
    else:
        new = torch.nn.Linear(*reversed(old.weight.shape), bias=True)
        with torch.no_grad():
            new.weight.copy_(2 * old.weight)
            new.bias.zero_()
        setattr(mlp, layer, new)
        factor = 2.0
    try:
        assert not tp.runs_plain(getattr(mlp, layer))
        y = mlp(x)
        y.sum().backward()
    finally:
        if handle is not None:
            handle.remove()
    w_up = old.weight if layer == "up" else mlp.up.weight
    w_down = old.weight if layer == "down" else mlp.down.weight
    f_up, f_down = (factor, 1.0) if layer == "up" else (1.0, factor)
    want = f_down * (ops.swiglu(f_up * x @ w_up.t()) @ w_down.t())
    assert torch.allclose(y, want, rtol=1e-5, atol=1e-6)
    if change.startswith("global") or change == "hook":
        assert old in seen


@pytest.mark.parametrize("kinds", ["qq", "kq", "kqq", "qkq", "kkqq", "kqkq", "qqqq"])
def test_flash_backward_accumulator_handover_orders_its_barriers(kinds):
    """The issuer and an epilogue warp of csrc/attention/flash_bwd.cu, in every interleaving, over the barriers acc (product finished) and
    accfree (read out) of the two accumulators.  A waiter sees the parity of a phase only, so a barrier must not complete a phase more
    while somebody still has to pass the last one; a shared phase count for both kinds (acc[1] committed by dQ items too, which waited for
    accfree[0] alone) breaks that."""
    def program(counted):
        issuer, epilogue, k, kv = [], [], 0, 0
        for kind in kinds:
            dkv = kind == "k"
            n = kv if counted else k                                    # the use of acc[1] / accfree[1]
            if dkv:
                issuer += ([("wait", "accfree0", k - 1)] if k else []) + [("done", "acc0")]
                issuer += ([("wait", "accfree1", n - 1)] if n else []) + [("done", "acc1")]
            else:
                issuer += ([("wait", "accfree0", k - 1)] if k else []) + [("done", "acc0")] + ([] if counted else [("done", "acc1")])
            epilogue += [("wait", "acc0", k), ("done", "accfree0")]
            if dkv or not counted:
                epilogue += [("wait", "acc1", n), ("done", "accfree1")]
            k, kv = k + 1, kv + dkv
        return issuer, epilogue

    def sound(programs):
        """Every reachable state: no waiter is a whole phase behind, nobody passes a wait early, both sides end."""
        seen, todo = set(), [((0, 0), ())]
        while todo:
            at, phases = state = todo.pop()
            if state in seen:
                continue
            seen.add(state)
            done, moved = dict(phases), False
            for i, ops in enumerate(programs):
                if at[i] == len(ops):
                    continue
                op = ops[at[i]]
                n = done.get(op[1], 0)
                if op[0] == "wait":
                    if n > op[2] + 1 or (n & 1 != op[2] & 1) != (n == op[2] + 1):
                        return False                                    # the parity no longer tells this phase from another
                    if n != op[2] + 1:
                        continue
                nxt = dict(done, **({op[1]: n + 1} if op[0] == "done" else {}))
                todo.append((tuple(a + (j == i) for j, a in enumerate(at)), tuple(sorted(nxt.items()))))
                moved = True
            if not moved and any(at[i] < len(programs[i]) for i in (0, 1)):
                return False
        return True

    assert sound(program(counted=True))
    assert sound(program(counted=False)) == ("q" not in kinds[1:])



def test_flash_backward_slots_follow_their_hand_backs(tmp_path):
    """csrc/attention/flash_bwd_slots.cuh against a queue of slots, over runs of items of 1 to 17 blocks: loads and hand-backs are numbered
    in their stated orders without gaps, a load takes the slot that was handed back first, and what lay there was handed back no later
    than the hand-back that the load waits for."""
    import shutil
    import subprocess
    root = Path(__file__).resolve().parents[1]
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    (tmp_path / "t.cpp").write_text(r"""
#define __device__
#define __forceinline__ inline
#include "attention/flash_bwd_slots.cuh"
#include <cstdio>
#include <cstdlib>
#include <tuple>
#include <map>
#include <vector>
using namespace llmctl::fbwd;
typedef std::tuple<char, int, int> Tile;                    // r or e, operand, block
#define CHECK(x) if (!(x)) { printf("line %d\n", __LINE__); return 1; }
int main() {
  srand(1);
  for (int run = 0; run < 200; ++run) {
    Slots s;
    std::vector<uint32_t> queue;                            // slots in the order in which they are free
    for (uint32_t i = 0; i < kTiles; ++i) queue.push_back(i);
    std::map<uint32_t, uint32_t> free_at;                   // slot -> number of the hand-back that freed it
    for (int item = 0; item < 40; ++item) {
      const int n = run % 4 ? 1 + rand() % 4 : 1 + rand() % 17;
      std::vector<Tile> loads, backs;
      for (int i = 0; i < n; ++i)
        for (int w = 0; w < 2; ++w) {
          if (i == 0) loads.push_back(Tile('r', w, 0));
          loads.push_back(Tile('e', w, i));
        }
      for (int i = 0; i < n; ++i) {
        if (n == 1) { backs.push_back(Tile('r', 0, 0)); backs.push_back(Tile('r', 1, 0)); }
        backs.push_back(Tile('e', 1, i));
        if (i == n - 2) backs.push_back(Tile('r', 0, 0));
        backs.push_back(Tile('e', 0, i));
        if (i == n - 2) backs.push_back(Tile('r', 1, 0));
      }
      auto slot = [&](Tile t) { return std::get<0>(t) == 'r' ? s.res(std::get<1>(t)) : s.streamed(std::get<1>(t), std::get<2>(t)); };
      size_t back = 0;
      for (size_t j = 0; j < loads.size(); ++j) {
        const Tile t = loads[j];
        const uint32_t l = s.base + j;
        CHECK((std::get<0>(t) == 'r' ? s.load_res(std::get<1>(t)) : s.load_streamed(std::get<1>(t), std::get<2>(t))) == l)
        while (queue.size() <= l) {                         // this item's own hand-backs, in order
          free_at[slot(backs[back])] = s.base + back;
          queue.push_back(slot(backs[back++]));
        }
        CHECK(slot(t) == queue[l])
        CHECK(l < kTiles || free_at[slot(t)] <= l - kTiles)
      }
      for (size_t j = 0; j < backs.size(); ++j) {
        const Tile t = backs[j];
        CHECK((std::get<0>(t) == 'r' ? s.given_res(std::get<1>(t), n) : s.given_streamed(std::get<1>(t), std::get<2>(t), n)) == s.base + j)
        if (j >= back) {
          free_at[slot(t)] = s.base + j;
          queue.push_back(slot(t));
        }
      }
      s.next(n);
    }
  }
  return 0;
}
""")
    subprocess.run([gxx, "-std=c++17", "-I", str(root / "csrc"), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("node", ["_LinearSwiGLUFn", "_SwiGLUMLPFn"])
def test_gated_backwards_write_within_their_gradient(monkeypatch, node):
    """gate | up that comes back from a hook on saved tensors as rows with gaps: the kernels have one row stride for it and for its gradient."""
    from types import SimpleNamespace
    from llmctl_b200.ops import functional as ops
    from llmctl_b200.ops import native
    rows, width, cols = 6, 16, 24
    gu = torch.zeros(rows, 2 * width + 8, dtype=torch.bfloat16)[:, :2 * width]
    x, up, down, act = (torch.zeros(*s, dtype=torch.bfloat16) for s in ((rows, 8), (2 * width, 8), (cols, width), (rows, width)))
    stride, operands = {}, []
    monkeypatch.setattr(native, "stream_ptr", lambda: 0)
    monkeypatch.setattr(native, "call", lambda name, *a: stride.update(gate_up=a[5] if name == "llmctl_swiglu_bwd" else a[9]))
    monkeypatch.setattr(ops, "gemm_raw", lambda a, b, **k: operands.append(a))
    monkeypatch.setattr(ops, "_wgrad", lambda *a: None)
    saved = (x, up, gu) if node == "_LinearSwiGLUFn" else (x, up, down, gu, act)
    ctx = SimpleNamespace(needs_input_grad=[True] * 3, saved_tensors=saved, kept_as=tuple((t.shape, t.dtype, t.device) for t in saved))
    getattr(ops, node).backward(ctx, act if node == "_LinearSwiGLUFn" else torch.zeros(rows, cols, dtype=torch.bfloat16))
    (dgu,) = operands
    assert dgu.stride(0) == stride["gate_up"] and dgu.untyped_storage().nbytes() >= 2 * ((rows - 1) * stride["gate_up"] + 2 * width)


@pytest.mark.parametrize("form", ["wider", "part", "as it was"])
@pytest.mark.parametrize("call", ["rmsnorm", "rmsnorm and sum", "layernorm", "rotation", "swiglu", "swiglu and product", "product", "product and swiglu", "mlp",
                                  "attention", "rotation and attention"])
def test_backwards_refuse_saved_tensors_of_other_forms(monkeypatch, call, form):
    """What a hook on saved tensors gives back is looked at before any kernel is called: its address says nothing of its type and size."""
    from llmctl_b200.ops import attention as attn
    from llmctl_b200.ops import functional as ops
    from llmctl_b200.ops import native
    calls = []
    monkeypatch.setattr(native, "stream_ptr", lambda: 0)
    monkeypatch.setattr(native, "has_symbol", lambda name: True)
    monkeypatch.setattr(native, "call", lambda name, *a: calls.append(name))
    monkeypatch.setattr(ops, "_scratch", lambda device, n, name: torch.zeros(n))

    def product(a, b, *, a_mn=False, b_mn=False, **k):
        calls.append("product")
        return torch.zeros(a.shape[int(a_mn)], b.shape[int(b_mn)], dtype=a.dtype)
    monkeypatch.setattr(ops, "gemm_raw", product)
    z = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, requires_grad=True)                # noqa: E731
    table = torch.zeros(8, 32)
    run = {"rmsnorm": lambda: ops._RMSNormFn.apply(z(6, 16), None, z(16), 1e-5)[0], "rmsnorm and sum": lambda: ops._RMSNormFn.apply(z(6, 16), z(6, 16), z(16), 1e-5)[0],
           "layernorm": lambda: ops._LayerNormFn.apply(z(6, 16), None, z(16), z(16), 1e-5)[0],
           "rotation": lambda: ops._RopeFn.apply(z(6, 128) * 1, table, table, 2, 64, 6, None), "swiglu": lambda: ops._SwiGLUFn.apply(z(6, 32)),
           "swiglu and product": lambda: ops._SwiGLULinearFn.apply(z(6, 32), z(8, 16)), "product": lambda: ops._LinearFn.apply(z(6, 16), z(8, 16)),
           "product and swiglu": lambda: ops._LinearSwiGLUFn.apply(z(6, 16), z(32, 16)), "mlp": lambda: ops._SwiGLUMLPFn.apply(z(6, 16), z(32, 16), z(8, 16)),
           "attention": lambda: attn._FlashAttnFn.apply(z(2, 6, 1, 64), z(2, 6, 1, 64), z(2, 6, 1, 64), 1.0, True),
           "rotation and attention": lambda: attn._RopeAttnPackedFn.apply(z(6, 192) * 1, table, table, 1, 6, 1, 64, None, 1.0, True)}[call]
    unpack = {"wider": torch.Tensor.double, "part": lambda t: t[:-1], "as it was": lambda t: t}[form]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        y = run()
    calls.clear()
    with contextlib.nullcontext() if form == "as it was" else pytest.raises(RuntimeError, match="came back"):
        y.backward(torch.zeros_like(y))
    assert bool(calls) == (form == "as it was")


def test_division_by_a_launch_constant(tmp_path):
    """csrc/common/fast_div.h against the machine's division: divisors and numbers at and around powers of two, the ends of their ranges,
    and a spread of others."""
    import shutil
    import subprocess
    root = Path(__file__).resolve().parents[1]
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    (tmp_path / "t.cpp").write_text(r"""
#include "common/fast_div.h"
#include <cstdio>
#include <random>
#include <vector>
int main() {
  std::mt19937 g(1);
  std::vector<uint32_t> some = {1, 3, 5, 7, 11, 40, 148, 185, 641, 65537, 0x7fffffffu};
  for (int b = 0; b < 31; ++b)
    for (int e = -1; e <= 1; ++e) some.push_back((1u << b) + e);
  for (int i = 0; i < 2000; ++i) some.push_back(g() >> (1 + g() % 30));
  for (uint32_t d : some) {
    if (d == 0) continue;
    const llmctl::FastDiv f(d);
    for (uint32_t n : some) {
      uint32_t rem;
      const uint32_t q = f.divide(n, rem);
      if (q != n / d || rem != n % d) { printf("%u / %u = %u rest %u\n", n, d, q, rem); return 1; }
    }
  }
  return 0;
}
""")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", str(root / "csrc"), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_items_of_the_attention_forward(tmp_path):
    """csrc/attention/flash_split.h takes the items that were measured to be at least 3% faster, from operands in L2 and in memory alike, at the sizes
    on either side of its lines."""
    import shutil
    import subprocess
    root = Path(__file__).resolve().parents[1]
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    # (head size, mask, heads): (key blocks where single tiles won, where pairs won)
    won = {(64, 1, 12): ([2, 3, 8, 16, 24, 32], []), (64, 1, 16): ([2, 3, 9, 16, 24], [32]), (64, 1, 24): ([2, 3, 7, 13, 14], [20, 24]),
           (64, 1, 32): ([2, 4, 5, 7, 9], [12, 20]), (64, 1, 48): ([2, 3, 4], [5, 8, 20]), (64, 1, 96): ([], [4, 6, 8]),
           (128, 1, 16): ([2, 3, 9, 16, 20], [32]), (128, 1, 20): ([2, 5, 10, 14], [20, 24]), (128, 1, 32): ([2, 4, 5, 6, 7, 8], [12, 14, 20]),
           (128, 1, 40): ([2, 4], [5, 7, 8, 10, 20]), (128, 1, 64): ([2], [3, 4, 8]), (128, 1, 80): ([], [2, 4, 8]), (128, 1, 128): ([], [2, 3, 4, 8]),
           (64, 0, 12): ([2, 4, 8, 12], [16]), (64, 0, 16): ([2, 4, 8], [10, 12]), (128, 0, 16): ([2, 4, 8], [10, 12]), (128, 0, 40): ([2, 3, 7], [4, 5, 6]),
           (128, 0, 128): ([], [2, 3, 4])}
    (tmp_path / "t.cpp").write_text("#include \"attention/flash_split.h\"\n#include <cstdio>\nint main() {\n" + "".join(
        f'  printf("%d", llmctl::split_keys({heads}, {n}, {dim}, {mask}, 148));\n' for (dim, mask, heads), sides in won.items() for n in sides[0] + sides[1]) + "}\n")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", str(root / "csrc"), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    got = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True).stdout
    assert got == "".join("1" * len(a) + "0" * len(b) for a, b in won.values())


def test_shared_memory_limits_are_raised_and_never_lowered(tmp_path):
    """csrc/common/smem_limit.h with the runtime's two calls replaced: threads that ask for unlike sizes of one kernel leave the largest in
    place, a device counts by itself, and a call that was refused is asked again."""
    import shutil
    import subprocess
    root = Path(__file__).resolve().parents[1]
    gxx, cuda = shutil.which("g++"), Path("/usr/local/cuda/include")
    if gxx is None or not (cuda / "cuda_runtime_api.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "t.cpp").write_text(r"""
#include "common/smem_limit.h"
#include <atomic>
#include <thread>
#include <vector>
#include <cstdio>
static thread_local int device = 0;
static std::atomic<int> limit[2], calls, refuse;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) {
  ++calls;
  if (refuse) return cudaErrorInvalidValue;
  limit[device] = v;
  return cudaSuccess;
}
static void kernel() {}
#define EXPECT(c) if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; }
int main() {
  using llmctl::allow_smem;
  EXPECT(allow_smem(kernel, 200) == cudaSuccess && limit[0] == 200);
  std::thread([] { allow_smem(kernel, 100); }).join();             // another thread's table is empty
  EXPECT(limit[0] == 200 && calls == 1);
  EXPECT(allow_smem(kernel, 200) == cudaSuccess && limit[0] == 200);
  device = 1;
  EXPECT(allow_smem(kernel, 100) == cudaSuccess && limit[1] == 100 && limit[0] == 200);
  refuse = 1;
  EXPECT(allow_smem(kernel, 300) == cudaErrorInvalidValue);
  refuse = 0;
  EXPECT(allow_smem(kernel, 300) == cudaSuccess && limit[1] == 300);
  device = 0;
  std::vector<std::thread> ts;
  std::atomic<int> bad{0};
  for (int i = 0; i < 8; ++i)
    ts.emplace_back([&, i] {
      for (int k = 0; k < 2000; ++k) {
        const int n = 201 + (k * 7 + i * 13) % 500;
        if (allow_smem(kernel, n) != cudaSuccess || limit[0] < n) ++bad;
      }
    });
  for (auto& t : ts) t.join();
  EXPECT(bad == 0 && limit[0] == 700);
}
""")
    exe = tmp_path / "t"
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", str(root / "csrc"), "-I", str(cuda), str(tmp_path / "t.cpp"), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout


@pytest.mark.parametrize("shift,grad,native_rows", [(0, True, True), (1, True, False), (4, True, False), (8, True, True), (1, False, True)])
def test_cross_entropy_of_rows_at_odd_addresses_stays_off_the_kernel(monkeypatch, shift, grad, native_rows):
    """The loss kernels read and write 16-byte units: logits that begin elsewhere take the library path, unless they are copied first."""
    from llmctl_b200.ops import functional as ops
    base = torch.randn(4 * 64 + 8).bfloat16().requires_grad_(grad)      # the allocator's boundaries are multiples of 64 bytes
    logits = base[shift:shift + 256].view(4, 64)
    assert logits.data_ptr() % 16 == 2 * shift % 16
    t = torch.tensor([1, -100, 63, 5])
    calls = []
    monkeypatch.setattr(ops, "_use_native", lambda *a: True)
    monkeypatch.setattr(ops._CrossEntropyFn, "apply", lambda x, *a: calls.append(x.data_ptr()) or torch.zeros(()))
    loss = ops.cross_entropy(logits, t)
    assert bool(calls) == native_rows and all(p % 16 == 0 for p in calls)
    if not native_rows:
        loss.backward()
        assert torch.equal(loss, torch.nn.functional.cross_entropy(logits.float(), t)) and base.grad is not None


def test_paged_decode_scratch_is_counted_in_64_bits():
    """256 sequences of 128 heads in 512 splits want more than 2^31 numbers: the entry point returns them as a long long."""
    from llmctl_b200.ops import native, serving
    if not native.available():
        pytest.skip("kernel library not built")
    for batch, heads, dim, splits in ((256, 128, 128, 512), (65535, 32, 128, 8), (16, 32, 128, 8), (1, 12, 64, 8), (700, 1, 64, 1)):
        one_wave = splits == 1 or (splits <= 8 and batch * heads * splits <= 3 * 148)
        want = 0 if one_wave else batch * heads * splits * (dim + 2)
        assert native.lib().llmctl_paged_attn_scratch_elems(batch, heads, dim, splits) == want


@pytest.mark.parametrize("byte,name", [(0, "flash attention forward"), (1, "flash attention backward"), (2, "cross-entropy"), (3, "latent attention")])
def test_waits_that_ran_out_are_raised_once_wherever_the_host_looks(monkeypatch, byte, name):
    """The word that kernels write when a wait runs out, faked: reported by name at a check and before the next launch, then cleared."""
    import ctypes
    from llmctl_b200.ops import native
    word, launched, cleared = ctypes.c_uint32(0), [], []
    monkeypatch.setattr(native, "_wait_word", word)
    monkeypatch.setattr(native, "_wait_bound", True)
    monkeypatch.setattr(native, "_functions", {"llmctl_x": lambda *a: launched.append(a) or 0,
                                               **{status: cleared.append for _, status in native._WAITS}})
    native.check_waits("nothing")
    native.call("llmctl_x", 1)
    word.value = 1 << 8 * byte
    with pytest.raises(native.NativeError, match=f"in: {name} \\(this step\\)"):
        native.check_waits("this step")
    assert word.value == 0 and cleared == [1, 1, 1, 1]
    native.check_waits("again")
    word.value = 1 << 8 * byte
    with pytest.raises(native.NativeError, match=name):
        native.call("llmctl_x", 2)
    native.call("llmctl_x", 3)
    assert launched == [(1,), (3,)]


def test_training_and_serving_report_waits_that_ran_out(monkeypatch, tmp_path):
    """A wait that ran out during a step ends training before the window is logged or a checkpoint is written, and a served step before its
    tokens are handed out."""
    import ctypes
    from llmctl_b200.comms import mesh
    from llmctl_b200.ops import native
    from llmctl_b200.runtime.engine import TrainingEngine, create_training_config
    from llmctl_b200.serve.engine import InferenceEngine
    mesh.reset_state()
    word = ctypes.c_uint32(0)
    monkeypatch.setattr(native, "_wait_word", word)
    eng = TrainingEngine(create_training_config(model_name_or_path="gpt-tiny", output_dir=str(tmp_path), batch_size=2, seq_len=16, max_steps=3,
                                                logging_steps=1, eval_steps=0, kernels="native"))
    step = eng.train_step
    monkeypatch.setattr(eng, "train_step", lambda: (step(), setattr(word, "value", 1 << 8))[0])
    with pytest.raises(native.NativeError, match="flash attention backward"):
        eng.train()
    assert eng.global_step == 1 and not list(tmp_path.rglob("*.safetensors"))
    word.value = 1
    with pytest.raises(native.NativeError, match="checkpoint"):
        eng.save_checkpoint()
    word.value = 1 << 16
    with pytest.raises(native.NativeError, match="evaluation"):
        eng.evaluate()
    serving = InferenceEngine("gpt-tiny", device="cpu", kv_block_size=4, num_kv_blocks=64)
    seq = serving.add_request([1, 2, 3], 4, 0.0, 1.0, -1)
    word.value = 1
    with pytest.raises(native.NativeError, match="tokens"):
        serving.step()
    assert seq.generated == []


# pairs of 512 / 513 and more: the splits of long contexts; 444 pairs (three CTAs on each of 148 SMs) / 445: one launch or the merge kernel
@pytest.mark.parametrize("batch,heads,dim,context,splits,launch", [
    (16, 32, 128, 4096, 8, 8), (16, 32, 128, 512, 3, 3), (19, 27, 128, 4096, 3, 3), (32, 32, 128, 4096, 2, 2), (32, 32, 128, 512, 2, 2),
    (64, 32, 128, 4096, 1, 1), (256, 32, 128, 4096, 1, 1), (64, 12, 64, 512, 2, 1), (64, 12, 64, 1024, 2, 2), (37, 12, 64, 768, 3, 1),
    (37, 12, 64, 769, 3, 3), (89, 5, 64, 768, 3, 3), (8, 4, 128, 2304, 36, 8), (1, 32, 128, 4096, 37, 8), (1, 32, 128, 8192, 37, 37),
    (4, 32, 128, 1024, 10, 3), (64, 4, 128, 512, 5, 1), (1, 1, 64, 10, 1, 1)])
def test_decode_splits_by_pairs_of_head_and_sequence(batch, heads, dim, context, splits, launch):
    from llmctl_b200.ops import serving
    assert serving.choose_splits(batch, heads, context, 16) == splits
    assert serving._launch_splits(batch, heads, dim, context, 16) == launch


@pytest.mark.parametrize("name,operands,tail", [
    ("llmctl_rmsnorm_fwd", ["x", "residual", "w", "h", "y", None], (4, 64, 1e-5, None)),
    ("llmctl_rmsnorm_bwd", ["dy", "h", "w", None, "dres", "dx", None, "scratch"], (4, 4, 64, 0, None)),
    ("llmctl_rmsnorm_bwd_noalloc", ["dy", "h", "w", None, "dres", "dx", None], (4, 64, 0, None)),
    ("llmctl_layernorm_fwd", ["x", "residual", "w", "b", "h", "y", None, None], (4, 64, 1e-5, None)),
    ("llmctl_layernorm_bwd", ["dy", "h", "w", None, None, "dres", "dx", None, None, "scratch"], (4, 4, 64, 0, None)),
    ("llmctl_swiglu_fwd", ["gate_up", "out"], (4, 64, 128, None)),
    ("llmctl_swiglu_bwd", ["dout", "gate_up", "d_gate_up"], (4, 64, 128, None)),
])
def test_entries_refuse_odd_addresses(name, operands, tail):
    """An operand that the kernels read or write in 16-byte units and that begins inside one is an invalid value (1), told before anything is
    launched."""
    from llmctl_b200.ops import native
    fn = getattr(native.ctypes.CDLL(str(native.library_path())), name)
    fn.argtypes = [native.c_void_p] * len(operands) + [native.c_float if isinstance(v, float) else native.c_void_p if v is None else native.c_ll for v in tail]
    for odd in (i for i, operand in enumerate(operands) if operand):
        at = [1 << 20] * len(operands)
        at[odd] += 2
        assert fn(*at, *tail) == 1, operands[odd]


def test_decode_gemm_scratch_belongs_to_a_stream(monkeypatch):
    """Partials and tickets of the decode GEMM: one pair per stream, grown where a call needs more, a bounded number of streams; captured calls take
    partials of their own and one set of zeroed tickets per capture."""
    from llmctl_b200.ops import functional as ops, native
    now = {"stream": 1, "capture": 0}

    class Lib:
        @staticmethod
        def llmctl_stream_capture_id(stream):
            return now["capture"]
    monkeypatch.setattr(ops, "_skinny_ws", {})
    monkeypatch.setattr(ops, "_skinny_captures", {})
    monkeypatch.setattr(native, "stream_ptr", lambda: now["stream"])
    monkeypatch.setattr(native, "lib", lambda: Lib)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: now["capture"] != 0)
    x = torch.empty(2, 8)

    def ask(stream, elems, capture=0):
        now.update(stream=stream, capture=capture)
        return ops._skinny_workspace(x, elems)
    a, b = ask(1, 1000), ask(2, 1000)
    assert ask(1, 2000)[0] is a[0] and ask(1, 2000)[1] is a[1]
    assert a[0] is not b[0] and a[1] is not b[1] and not a[1].any() and a[1].dtype == torch.int32
    grown = ask(1, (1 << 20) + 1)
    assert grown[0].numel() > 1 << 20 and grown[1] is a[1] and ask(1, 5)[0] is grown[0]
    assert ask(1, 1 << 40)[0].numel() == ops._SKINNY_ELEMS                     # too few: the kernel takes whole tiles
    first, again, other, elsewhere = ask(1, 1000, 7), ask(1, 1000, 7), ask(1, 1000, 8), ask(2, 1000, 8)
    assert first[1] is again[1] and first[0] is not again[0]
    assert len({id(t[1]) for t in (first, other, elsewhere, grown, b)}) == 5
    assert ask(1, 1000)[1] is a[1] and ask(2, 1000)[1] is b[1]
    for stream in range(3, 40):
        ask(stream, 10)
    assert len(ops._skinny_ws) == ops._SKINNY_STREAMS and (x.get_device(), 39) in ops._skinny_ws and (x.get_device(), 1) not in ops._skinny_ws
    assert ops._skinny_workspace(x, 10, 39)[1] is ask(39, 10)[1]


@pytest.mark.parametrize("M,N,K,splits,elems", [(1, 128, 64, 0, 1 * 2 * 16 * 128), (17, 129, 4096, 0, 2 * 9 * 32 * 128), (16, 4096, 4096, 4, 32 * 5 * 16 * 128),
                                                (32, 12288, 4096, 0, 96 * 3 * 32 * 128)])
def test_decode_gemm_scratch_size(M, N, K, splits, elems):
    """tiles x (most CTAs that share one) x rows of the tile's width x 128."""
    from llmctl_b200.ops import native
    assert native.lib().llmctl_gemm_skinny_scratch_elems(M, N, K, splits) == elems


def test_cache_entries_refuse_odd_addresses():
    """As above for the append to the paged cache (packed rows, both caches) and the decode over it (queries read in pairs, both caches)."""
    from llmctl_b200.ops import native
    lib = native.ctypes.CDLL(str(native.library_path()))
    p, i, ll, f = native.c_void_p, native.c_int, native.c_ll, native.c_float
    lib.llmctl_kv_append.argtypes = [p, ll, i, i, p, p, p, i, i, i, p]
    lib.llmctl_paged_attn_decode.argtypes = [p, ll, p, p, p, i, p, p, ll, p, i, i, i, i, i, i, f, p]
    at = 1 << 20
    for odd in ((2, 0, 0), (0, 2, 0), (0, 0, 8)):
        assert lib.llmctl_kv_append(at + odd[0], 384, 128, 256, at + odd[1], at + odd[2], at, 2, 2, 64, None) == 1
        assert lib.llmctl_paged_attn_decode(at + odd[0], 128, at + odd[1], at + odd[2], at, 4, at, at, 128, None, 2, 2, 64, 16, 64, 1, 0.125, None) == 1


def test_dependent_kernels_wait_before_they_leave():
    """csrc/common/dependent.cuh, rule 1: a kernel that is launched beside the end of the one before it waits for that one on every way out
    and before it lets its own dependents in, or the order of the stream is lost for those behind it."""
    import re
    seen = []
    for path in sorted((Path(__file__).resolve().parents[1] / "csrc").rglob("*.cu")):
        text = path.read_text()
        bodies = {}
        for m in re.finditer(r"__global__ void (?:__\w+__\([^)]*\) )*\s*(\w+)\(", re.sub(r"\s*\n\s*", lambda m: " " * len(m.group()), text)):
            bodies[m.group(1)] = text[text.index(") {", m.end()):text.index("\n}", m.end())]
        launched = set(re.findall(r"launch_dependent\((\w+_kernel)\b", text))
        for name, body in bodies.items():
            wait = re.search(r"\bwait_for_previous\(", body)
            if wait is None:
                assert name not in launched, f"{path.name}: {name}"
                continue
            seen.append(name)
            for leaving in (r"\breturn;", r"\brelease_dependents\("):
                first = re.search(leaving, body)
                assert first is None or wait.start() < first.start(), f"{path.name}: {name}: {first.group()} before the wait"
    assert len(seen) >= 18 and {"flash_bwd_kernel", "gemm2_tcgen05_kernel", "norm_bwd_kernel", "paged_attn_decode_kernel"} <= set(seen), seen


def test_operator_extension_is_not_a_condition(monkeypatch, tmp_path):
    """An extension that is missing, no library at all or of another PyTorch leaves the Python operators in place, and says so."""
    import sys
    from llmctl_b200.ops import native
    built = native._OPS_PATH
    monkeypatch.setattr(native, "_OPS_PATH", tmp_path / "llmctl_ops.so")
    monkeypatch.setattr(native, "fast", native._NoOps())

    def left_out(why):
        with pytest.warns(RuntimeWarning, match=why):
            native._load_ops()
        assert native.fast.rmsnorm(1, 2) is None and native.fast.launches() == 0
    left_out("not built")
    native._OPS_PATH.write_text("x")
    left_out("not used")
    if built.exists():
        monkeypatch.setattr(native, "_OPS_PATH", built)
        monkeypatch.setattr(torch, "__version__", "0.0.1")
        left_out(f"this is PyTorch 0.0.1 and Python 3.{sys.version_info[1]}")


def test_has_symbol_tells_a_missing_entry_from_a_library_that_does_not_load(monkeypatch):
    from llmctl_b200.ops import native
    monkeypatch.setattr(native, "_lib", None)
    monkeypatch.setattr(native, "_functions", {})

    def failing(error):
        def lib():
            raise error
        return lib
    for built in (True, False):
        monkeypatch.setattr(native, "available", lambda: built)
        for error in (OSError("no loader"), RuntimeError("not this one")):
            monkeypatch.setattr(native, "lib", failing(error))
            if built:
                with pytest.raises(type(error)):
                    native.has_symbol("llmctl_rmsnorm_fwd")
            else:
                assert not native.has_symbol("llmctl_rmsnorm_fwd")
    monkeypatch.setattr(native, "available", lambda: True)
    monkeypatch.setattr(native, "lib", lambda: type("Library", (), {"llmctl_rmsnorm_fwd": 1}))
    assert native.has_symbol("llmctl_rmsnorm_fwd") and not native.has_symbol("llmctl_rmsnorm_bwd")


def test_build_of_the_operator_extension(monkeypatch, tmp_path):
    """It is built with the whole library and where it was built before, not for a part of the kernels, and again for another PyTorch."""
    import importlib.util
    spec = importlib.util.spec_from_file_location("build_native_under_test", Path(__file__).resolve().parents[1] / "build_native.py")
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    lib, src = tmp_path / "llmctl_ops.so", tmp_path / "ops.cpp"
    monkeypatch.setattr(b, "LIBDIR", tmp_path)
    monkeypatch.setattr(b, "CSRC", tmp_path)
    monkeypatch.setattr(b, "_component_sources", lambda components: [])
    monkeypatch.setattr(b, "_build_operators", lambda *a: lib)
    assert "operators" not in b.build(components=["serve"]) and "operators" not in b.build(operators=False)
    assert b.build()["operators"] == b.build(components=["all"])["operators"] == b.build(components=["serve"], operators=True)["operators"] == str(lib)
    monkeypatch.setattr(b, "_operators_missing", lambda: "PyTorch")
    assert "PyTorch" in b.build()["operators"]
    src.write_text("")
    lib.write_text("")
    assert "operators" in b.build(components=["serve"])
    now = src.stat().st_mtime
    import os
    os.utime(lib, (now + 10, now + 10))
    assert not b._operators_current(lib, src, now)
    lib.with_suffix(".built").write_text(b._operators_stamp())
    assert b._operators_current(lib, src, now) and not b._operators_current(lib, src, now + 20)
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert not b._operators_current(lib, src, now)


def test_scratch_of_a_captured_call_is_its_own(monkeypatch):
    """Graphs captured on one stream may be replayed beside each other: they share no buffer, with each other or with that stream's calls."""
    from llmctl_b200.ops import functional as ops, native
    capturing = [False]
    monkeypatch.setattr(ops, "_scratch_cache", {})
    monkeypatch.setattr(native, "stream_ptr", lambda: 1)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    kept = ops._scratch(torch.device("cpu"), 100, "norm")
    assert ops._scratch(torch.device("cpu"), 50, "norm") is kept and ops._scratch(torch.device("cpu"), 50, "other") is not kept
    capturing[0] = True
    a, b = ops._scratch(torch.device("cpu"), 100, "norm"), ops._scratch(torch.device("cpu"), 100, "norm")
    assert a is not kept and b is not kept and a is not b
    capturing[0] = False
    assert ops._scratch(torch.device("cpu"), 100, "norm") is kept
