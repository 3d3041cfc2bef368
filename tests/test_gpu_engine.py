"""GPU end-to-end: fused executor against dense attention, and a tiny-model training step whose
gradients are compared with the same model evaluated with plain PyTorch ops in fp32."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")


def test_fused_executor_single_gpu():
    _need_gpu()
    res = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "fused_worker.py")], stdout=subprocess.PIPE,
                         stderr=subprocess.STDOUT, text=True, timeout=900, env=dict(os.environ, PYTHONPATH=ROOT))
    assert res.returncode == 0 and "FUSED_OK" in res.stdout, res.stdout[-3000:]


@pytest.mark.parametrize("world", [2, 4, 8])
def test_fused_executor_multi_gpu(world):
    """The fused executor on 2 / 4 / 8 GPUs against dense attention: peer operand fetch inside the
    kernels, partial (out, lse) stores into owners' arenas, merge, gradient push, flag barriers."""
    _need_gpu()
    if torch.cuda.device_count() < world:
        pytest.skip(f"needs {world} GPUs")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={world}", "--master-addr",
           "127.0.0.1", "--master-port", str(29541 + world), os.path.join(ROOT, "tests", "fused_worker.py")]
    # also exercises the executor's debugging modes: a status check after every phase, and staging
    # regions filled with a sentinel before every call (an un-fetched block would wreck the result)
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900,
                         env=dict(os.environ, PYTHONPATH=ROOT, DCP_B200_SYNCHRONOUS="1", DCP_B200_POISON="1"))
    assert res.returncode == 0 and "FUSED_OK" in res.stdout, res.stdout[-3000:]


def test_fused_executor_two_gpus_over_ipc_mapped_memory():
    """The second peer-memory route: arenas allocated by the in-tree library and mapped into the
    peer through CUDA IPC handles instead of the framework's symmetric-memory module."""
    _need_gpu()
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr",
           "127.0.0.1", "--master-port", "29553", os.path.join(ROOT, "tests", "fused_worker.py")]
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900,
                         env=dict(os.environ, PYTHONPATH=ROOT, DCP_B200_PEER_MEMORY="ipc"))
    assert res.returncode == 0 and "FUSED_OK" in res.stdout, res.stdout[-3000:]


def test_overlapped_sharded_optimizer_two_gpus():
    """Bucketed reduce-scatter on a side stream + sharded AdamW + all-gather against fp32
    torch.optim.AdamW on the rank-summed gradients, parameter rebuild from the master shards, and
    the status guard that keeps a detected failure away from the weights."""
    _need_gpu()
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr",
           "127.0.0.1", "--master-port", "29561", os.path.join(ROOT, "tests", "opt_worker.py")]
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=600,
                         env=dict(os.environ, PYTHONPATH=ROOT))
    assert res.returncode == 0 and "OPT_OK" in res.stdout, res.stdout[-3000:]


def test_tensor_parallel_step_two_gpus():
    """Tensor parallelism (heads and FFN split over two ranks): loss and gradients match the fp32
    model assembled from the shards; replicated parameters stay identical through a step."""
    _need_gpu()
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr",
           "127.0.0.1", "--master-port", "29547", os.path.join(ROOT, "tests", "tp_worker.py")]
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900,
                         env=dict(os.environ, PYTHONPATH=ROOT))
    assert res.returncode == 0 and "TP_OK" in res.stdout, res.stdout[-3000:]


def test_head_and_embedding_gradients_reach_autograd():
    """With hand-written layers the gradients of the embedding and the LM head still answer ``torch.autograd.grad``,
    tensor hooks, a ``.grad`` that is not there and one replaced before the backward; writing them directly gives the
    same (the embedding sums fp32 in another order and rounds to bf16 once: 2^-7 of the largest element)."""
    _need_gpu()
    from dcp_b200.data import synth
    from dcp_b200.models.llama import tiny_config
    from dcp_b200.train import EngineConfig, TrainEngine
    eng = TrainEngine(EngineConfig(tiny_config(n_layers=1, hidden=1024, n_heads=8, n_kv_heads=2, ffn=2048, vocab=512), tokens_per_step=512,
                                   block_size=256, length_dist=synth.LengthDist("lognormal", 200.0, 0.6, 64, 512), planner_workers=0,
                                   activation_budget_gb=0.0), torch.device("cuda", 0))
    model, plan = eng.model, eng.plans.get(0)
    assert model.layer_levels is not None
    inputs = (*eng.stage_inputs(plan), 1.0 / plan.n_global_tokens)
    pair = [model.p["embed"], model.p["lm_head"]]
    want = [g.float() for g in torch.autograd.grad(model.loss(*inputs), pair)]
    assert all(w.abs().max() > 0 for w in want)

    def check(grads):
        for g, w in zip(grads, want):
            assert (g.float() - w).abs().max() <= 2.0 ** -7 * w.abs().max()

    for write in (False, True):
        model.zero_grad()
        loss = model.loss(*inputs, write_grads=write)
        old, new = [t.grad for t in pair], [torch.zeros_like(t) for t in pair]
        for t, g in zip(pair, new):
            t.grad = g
        loss.backward()
        check(new)
        assert all(t.grad is g for t, g in zip(pair, new)) and all(not g.any() for g in old)
        for t in pair:
            t.grad = None
        model.loss(*inputs, write_grads=write).backward()
        check([t.grad for t in pair])
        seen = []
        handles = [t.register_hook(lambda g, i=i: seen.append(i)) for i, t in enumerate(pair)]
        handles += [t.register_post_accumulate_grad_hook(lambda t, i=i: seen.append(2 + i)) for i, t in enumerate(pair)]
        for t, g in zip(pair, old):
            t.grad = g
        model.loss(*inputs, write_grads=write).backward()
        assert sorted(seen) == [0, 1, 2, 3]
        check([t.grad for t in pair])
        for h in handles:
            h.remove()
    eng.close()


@pytest.mark.parametrize("layer_path", ["autograd", "level0", "level1+2", "auto"])
def test_tiny_model_step_matches_pytorch(layer_path):
    """Every layer implementation (autograd + checkpoint, hand-written backward at each activation
    level) must give the gradients of the fp32 PyTorch model."""
    _need_gpu()
    from dcp_b200.data import synth
    from dcp_b200.models.llama import tiny_config
    from dcp_b200.models.reference import reference_loss
    from dcp_b200.train import EngineConfig, TrainEngine
    dev = torch.device("cuda", 0)
    cfg = EngineConfig(tiny_config(n_layers=2, hidden=1024, n_heads=8, n_kv_heads=2, ffn=2048, vocab=2048),
                       tokens_per_step=1536, block_size=256,
                       length_dist=synth.LengthDist("lognormal", 400.0, 0.6, 64, 1536), planner_workers=0,
                       clip_grad=None,
                       activation_budget_gb={"autograd": -1.0, "level0": 0.0, "level1+2": 0.0, "auto": None}[layer_path])
    eng = TrainEngine(cfg, dev)
    if layer_path == "autograd":
        assert eng.model.layer_levels is None
    elif layer_path == "level0":
        assert eng.model.layer_levels == [0, 0]
    elif layer_path == "level1+2":
        eng.model.layer_levels = [1, 2]
    else:
        assert eng.model.layer_levels == [2, 2]     # a tiny model fits entirely
    plan = eng.plans.get(0)
    toks, labels, pos = eng.stage_inputs(plan)
    eng.model.zero_grad()
    loss = eng.model.loss(toks, labels, pos, 1.0 / plan.n_global_tokens)
    loss.backward()
    torch.cuda.synchronize()
    eng.executor.check_status()
    params32 = {k: v.detach().float().requires_grad_(True) for k, v in eng.model.p.items()}
    ref = reference_loss(eng.cfg.model, params32, toks, labels, pos, plan.seqlens, 1.0 / plan.n_global_tokens)
    ref.backward()
    assert abs(loss.item() - ref.item()) / abs(ref.item()) < 2e-2
    for name in ("l0.wqkv", "l1.wo", "l0.wgu", "l1.wd", "l0.norm1", "norm_f", "lm_head", "embed"):
        g, r = eng.model.p[name].grad.float(), params32[name].grad
        denom = r.abs().max() + 1e-6
        assert (g - r).abs().max() / denom < 8e-2, name
    l2 = eng.train_step(eng.plans.get(1))
    assert l2 == l2
    eng.close()


def test_checkpoint_resume_continues_identically(tmp_path):
    """Save after two steps, resume in a fresh engine: the third step's loss equals the loss of the
    engine that kept running (optimizer shards, bf16 parameters, iteration counter, batch order)."""
    _need_gpu()
    from dcp_b200.data import synth
    from dcp_b200.models.llama import tiny_config
    from dcp_b200.train import EngineConfig, TrainEngine
    dev = torch.device("cuda", 0)
    mk = lambda: TrainEngine(EngineConfig(tiny_config(n_layers=2, hidden=1024, n_heads=8, n_kv_heads=2, ffn=2048, vocab=2048),
                                          tokens_per_step=1536, block_size=256,
                                          length_dist=synth.LengthDist("lognormal", 400.0, 0.6, 64, 1536),
                                          planner_workers=0, lr=1e-3), dev)
    a = mk()
    a.train_step(); a.train_step()
    a.save_checkpoint(str(tmp_path))
    want = a.train_step()
    b = mk()
    b.load_checkpoint(str(tmp_path))
    assert b.iteration == 2
    got = b.train_step()
    assert abs(got - want) <= 1e-5 * max(1.0, abs(want)), (got, want)
    a.close(); b.close()


def test_checkpoint_written_by_two_ranks_resumes_on_one(tmp_path):
    """Resume on another number of GPUs: two ranks train two steps and save; one engine loads the
    files, re-cuts the sharded fp32 optimizer state and rebuilds exactly the bf16 parameters that
    the two ranks held, then trains on."""
    _need_gpu()
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr",
           "127.0.0.1", "--master-port", "29567", os.path.join(ROOT, "tests", "ckpt_worker.py"), str(tmp_path)]
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=600,
                         env=dict(os.environ, PYTHONPATH=ROOT))
    assert res.returncode == 0 and "CKPT_OK" in res.stdout, res.stdout[-3000:]
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    from ckpt_worker import engine_config
    from dcp_b200.train import TrainEngine
    dev = torch.device("cuda", 0)
    eng = TrainEngine(engine_config(), dev)
    eng.load_checkpoint(str(tmp_path))
    saved = torch.load(os.path.join(str(tmp_path), "rank000.pt"), map_location=dev, weights_only=False)
    assert eng.iteration == 2 and eng.optimizer.step_count == saved["optimizer"]["step"]
    assert torch.equal(eng.bufs.params, saved["params_bf16"])
    loss = eng.train_step()
    assert loss == loss
    eng.close()


def test_loss_trajectory_matches_fp32_pytorch_training():
    """Convergence equivalence (the reference overlays the loss curves of its runs, benchmark/plotting/
    plot_loss_curve.py): 20 optimizer steps on one fixed batch through the engine (bf16 kernels, fused
    attention, sharded AdamW) against the same model trained with plain fp32 PyTorch ops and
    torch.optim.AdamW.  Both losses must fall and the curves must lie on top of each other."""
    _need_gpu()
    from dcp_b200.data import synth
    from dcp_b200.models.llama import tiny_config
    from dcp_b200.models.reference import reference_loss
    from dcp_b200.train import EngineConfig, TrainEngine
    dev = torch.device("cuda", 0)
    cfg = EngineConfig(tiny_config(n_layers=2, hidden=1024, n_heads=8, n_kv_heads=2, ffn=2048, vocab=2048),
                       tokens_per_step=1536, block_size=256, length_dist=synth.LengthDist("lognormal", 400.0, 0.6, 64, 1536),
                       planner_workers=0, lr=3e-4, weight_decay=0.1, clip_grad=1.0)
    eng = TrainEngine(cfg, dev)
    plan = eng.plans.get(0)
    params32 = {k: v.detach().float().clone().requires_grad_(True) for k, v in eng.model.p.items()}
    ref_opt = torch.optim.AdamW(list(params32.values()), lr=3e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    ours, theirs = [], []
    for _ in range(20):
        toks, labels, pos = eng.stage_inputs(plan)
        ref_opt.zero_grad()
        ref = reference_loss(eng.cfg.model, params32, toks, labels, pos, plan.seqlens, 1.0 / plan.n_global_tokens)
        ref.backward()
        torch.nn.utils.clip_grad_norm_(list(params32.values()), 1.0)
        ref_opt.step()
        theirs.append(ref.item())
        ours.append(float(eng.run_step(toks, labels, pos, plan.n_global_tokens).item()))
    eng.check_status()
    eng.close()
    assert ours[-1] < 0.75 * ours[0] and theirs[-1] < 0.75 * theirs[0], (ours, theirs)
    # step by step within 3 % while the curves are steep (the first ten steps), and never further apart
    # than 5 % of the initial loss (a fixed batch is memorised quickly; tiny losses drift in bf16)
    early = max(abs(a - b) / abs(b) for a, b in zip(ours[:10], theirs[:10]))
    late = max(abs(a - b) for a, b in zip(ours, theirs)) / theirs[0]
    assert early < 3e-2 and late < 5e-2, (early, late, ours, theirs)


def test_training_from_the_dataloader_resumes_mid_epoch(tmp_path):
    """Dataset -> token-budget batch sampler -> planning dataloader -> TrainEngine.train_step: three
    steps from a synthetic corpus, a checkpoint after the second; a fresh engine that loads it and
    re-opens the dataloader continues with the third batch (sampler position is part of the
    checkpoint) and reproduces the third loss."""
    _need_gpu()
    from dcp_b200.data import synth
    from dcp_b200.models.llama import tiny_config
    from dcp_b200.train import EngineConfig, TrainEngine, dataset_batches
    dev = torch.device("cuda", 0)
    dist_ = synth.LengthDist("lognormal", 400.0, 0.6, 64, 1536)
    mk = lambda: TrainEngine(EngineConfig(tiny_config(n_layers=2, hidden=1024, n_heads=8, n_kv_heads=2, ffn=2048, vocab=2048),
                                          tokens_per_step=2048, block_size=256, length_dist=dist_, planner_workers=0,
                                          lr=1e-3), dev)
    a = mk()
    it_a = dataset_batches(a, 64, dist_)
    l1 = a.train_step(next(it_a)); l2 = a.train_step(next(it_a))
    assert a.samples_consumed > 0 and l1 == l1 and l2 == l2
    a.save_checkpoint(str(tmp_path))
    want = a.train_step(next(it_a))
    b = mk()
    b.load_checkpoint(str(tmp_path))
    assert b.samples_consumed == a.samples_consumed - len(a.last_seqlens)
    got = b.train_step(next(dataset_batches(b, 64, dist_)))
    assert abs(got - want) <= 1e-5 * max(1.0, abs(want)), (got, want)
    it_a.close()
    a.close(); b.close()


@pytest.mark.parametrize("impl", ["fused", "fused-from-plan-bytes"])
def test_reference_api_with_fused_backend(impl):
    """The reference's call sequence (get_executor(...), DCPAttention.apply) with the fused executor,
    its tables lowered from the placed workload or from plans deserialised from bytes: same local
    layouts as the plan interpreter, results equal to dense attention."""
    _need_gpu()
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.runtime.interface import DCPAttention, prepare_dcp_distributed_attn_for_test
    from dcp_b200.runtime.simulate import dense_reference
    dev = torch.device("cuda", 0)
    ctx = get_default_execution_context(1, 1)
    raw = [700, 300, 1100]
    ex, lq, lkv, ldo, q, kv, dout, _, pad = prepare_dcp_distributed_attn_for_test(
        raw, 8, 2, 128, 256, 8, ctx, 0, "lambda", torch.bfloat16, device=dev, executor_impl=impl)
    lq.requires_grad_(True); lkv.requires_grad_(True)
    out = DCPAttention.apply(ex, False, False, lq, lkv)
    out.backward(ldo)
    torch.cuda.synchronize()
    ex.impl.check_status()
    from dcp_b200.planner import masks
    m = masks.get_mask_fn("lambda")(raw, pad, torch.int32)
    ro, _, rdq, rdkv = dense_reference(q.float(), kv.float(), raw, pad, m, 128 ** -0.5, dout.float())
    rel = lambda a, b: ((a.float().cpu() - b).abs().max() / (b.abs().max() + 1e-9)).item()
    # one device, one head block: local order == global order
    assert rel(out.detach(), ro) < 3e-2 and rel(lq.grad, rdq) < 3e-2 and rel(lkv.grad, rdkv) < 3e-2
    assert set(ex.log_memory_usage()) >= {"q", "kv", "dq", "dkv"}


def test_program_tables_may_be_on_the_gpu_already():
    """``prepare`` takes a program whose tables were moved to the device before: the same results."""
    _need_gpu()
    import dataclasses
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.runtime.interface import DCPAttention, prepare_dcp_distributed_attn_for_test
    dev = torch.device("cuda", 0)
    ex, lq, lkv, *_ = prepare_dcp_distributed_attn_for_test([300, 129], 4, 2, 128, 256, 4, get_default_execution_context(1, 1), 0, "causal",
                                                            torch.bfloat16, device=dev, executor_impl="fused")
    want = DCPAttention.apply(ex, False, False, lq, lkv)
    p = ex.impl.program
    moved = dataclasses.replace(p, fwd=[t.to(dev) for t in p.fwd], bwd=[t.to(dev) for t in p.bwd])
    ex.impl.prepare(moved)
    assert torch.equal(DCPAttention.apply(ex, False, False, lq, lkv), want)


@pytest.mark.parametrize("head_dim,dtype", [(64, torch.float16), (96, torch.bfloat16), (128, torch.float32)])
def test_fused_backend_other_head_dims_and_dtypes(head_dim, dtype):
    """Head dimensions below 128 run zero-padded on the 128-channel kernels and fp16 / fp32 tensors
    are converted on the way in and out: results equal dense attention of the same inputs with the
    softmax scale of the real head dimension, in the caller's shapes and dtype."""
    _need_gpu()
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.planner import masks
    from dcp_b200.runtime.interface import DCPAttention, prepare_dcp_distributed_attn_for_test
    from dcp_b200.runtime.simulate import dense_reference
    dev = torch.device("cuda", 0)
    ctx = get_default_execution_context(1, 1)
    raw = [500, 1300, 260]
    ex, lq, lkv, ldo, q, kv, dout, _, pad = prepare_dcp_distributed_attn_for_test(
        raw, 8, 2, head_dim, 256, 8, ctx, 0, "causal", dtype, device=dev, executor_impl="fused")
    lq.requires_grad_(True); lkv.requires_grad_(True)
    out = DCPAttention.apply(ex, False, False, lq, lkv)
    out.backward(ldo)
    torch.cuda.synchronize()
    ex.impl.check_status()
    assert out.dtype == dtype and out.shape[-1] == head_dim and lq.grad.shape == lq.shape and lkv.grad.shape == lkv.shape
    m = masks.get_mask_fn("causal")(raw, pad, torch.int32)
    ro, _, rdq, rdkv = dense_reference(q.float(), kv.float(), raw, pad, m, head_dim ** -0.5, dout.float())
    rel = lambda a, b: ((a.float().cpu() - b).abs().max() / (b.abs().max() + 1e-9)).item()
    errs = (rel(out.detach(), ro), rel(lq.grad, rdq), rel(lkv.grad, rdkv))
    assert max(errs) < 3e-2, errs


@pytest.mark.parametrize("head_dim,dtype", [(128, torch.bfloat16), (64, torch.float32)])
def test_dcp_attention_reads_any_layout_and_keeps_calls_apart(head_dim, dtype):
    """Operands that the kernels can read in place, strided and misaligned ones give the same output bit for bit, and
    a second call before the first one's backward disturbs neither: all gradients are those of calls on their own.
    dQ is a sum of fp32 whose order may differ: 1e-5 of the largest element, and one bf16 rounding (2^-7 of the element)."""
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.runtime.interface import DCPAttention, prepare_dcp_distributed_attn_for_test
    dev = torch.device("cuda", 0)
    ex, lq, lkv, ldo, *_ = prepare_dcp_distributed_attn_for_test([300, 129], 4, 2, head_dim, 256, 4, get_default_execution_context(1, 1),
                                                                 0, "causal", dtype, 3, device=dev, executor_impl="fused")

    def call(q, kv):
        q, kv = q.detach().requires_grad_(True), kv.detach().requires_grad_(True)
        return q, kv, DCPAttention.apply(ex, False, False, q, kv)

    def grads(q, kv, out, do):
        res = torch.autograd.grad(out, (q, kv), do)
        assert all(g.dtype == dtype and g.shape == t.shape for g, t in zip(res, (q, kv)))
        return (out.detach(), *res)

    def same(got, want):
        assert torch.equal(got[0], want[0])
        for a, b in zip(got[1:], want[1:]):
            a, b = a.float(), b.float()
            ulp = 2.0 ** -7 if dtype == torch.bfloat16 else 0.0
            assert ((a - b).abs() <= ulp * b.abs() + 1e-5 * b.abs().max()).all()

    strided = lambda t: torch.stack([t, t * 2], dim=-1)[..., 0]
    shifted = lambda t: torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)
    second = (lq * 0.5, lkv + 1)
    alone, alone2 = grads(*call(lq, lkv), ldo), grads(*call(*second), torch.ones_like(ldo))
    assert (alone[1].float() - alone2[1].float()).abs().max() > 0.1 * alone[1].float().abs().max()
    for how in (lambda t: t, strided, shifted):
        q, kv, do = (how(t.clone()) for t in (lq, lkv, ldo))
        mine, other = call(q, kv), call(*second)
        same(grads(*mine, do), alone)
        same(grads(*other, torch.ones_like(ldo)), alone2)


class _Recorder:
    """The native calls of a program, and whether each call was taken."""

    def __init__(self, native):
        assert native is not None
        self.native, self.taken = native, []

    def _call(self, name, args):
        res = getattr(self.native, name)(*args)
        self.taken.append(res is not None)
        return res

    def __getattr__(self, name):       # the calls below the conversions
        return getattr(self.native, name)

    def forward(self, *args):
        return self._call("forward", args)

    def backward(self, *args):
        return self._call("backward", args)


@pytest.mark.parametrize("head_dim,dtype,kv_dtype", [(128, torch.bfloat16, None), (128, torch.float16, None), (72, torch.bfloat16, None),
                                                     (64, torch.float32, None), (24, torch.float32, None), (40, torch.float16, None),
                                                     (128, torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("form", ["rows", "flat", "strided", "halves"])
def test_native_calls_against_the_general_path(head_dim, dtype, kv_dtype, form):
    """The same call with its host side in native code and in Python: same output bits, types and shapes, and gradients
    that differ by the order of fp32 sums only (1e-5 of the largest, and one rounding of the result type).  The native code takes
    contiguous operands of one type; others go the general way from inside the call.  A wrong number of elements is refused by
    both."""
    _need_gpu()
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.ops import _lib
    from dcp_b200.runtime.interface import DCPAttention, prepare_dcp_distributed_attn_for_test
    dev = torch.device("cuda", 0)
    ex, lq, lkv, ldo, *_ = prepare_dcp_distributed_attn_for_test([300, 129], 4, 2, head_dim, 256, 4, get_default_execution_context(1, 1),
                                                                 0, "causal", dtype, 3, device=dev, executor_impl="fused")
    lkv = lkv.to(kv_dtype or dtype)
    native = _Recorder(ex.impl.native())
    how = {"rows": lambda t: t, "flat": lambda t: t.flatten(1), "strided": lambda t: torch.stack([t, t], -1)[..., 0],
           "halves": lambda t: t.flatten(0, 1).view(2, -1)}[form]

    def call(with_native):
        ex.impl._native = native if with_native else None
        before, launches = _lib.LAUNCHES, ex.impl.kernel_launches
        q, kv = how(lq.clone()).requires_grad_(True), how(lkv.clone()).requires_grad_(True)
        out = DCPAttention.apply(ex, False, False, q, kv)
        grads = torch.autograd.grad(out, (q, kv), ldo.to(out.dtype).view(out.shape))
        torch.cuda.synchronize()
        ex.impl.check_status()
        assert grads[0].shape == q.shape and grads[1].shape == kv.shape
        return (out.detach(), *grads), (_lib.LAUNCHES - before, ex.impl.kernel_launches - launches)

    (got, counted), (want, counted_too) = call(True), call(False)
    assert native.taken == [form != "strided" and kv_dtype is None] * 2     # forward, backward
    assert counted[1] == counted_too[1]
    if native.taken[0] and not (head_dim == 128 and dtype == torch.bfloat16):
        assert counted[0] < counted_too[0]                                  # conversions are part of other launches there
    else:
        assert counted[0] == counted_too[0]
    assert all(a.dtype == b.dtype and a.shape == b.shape for a, b in zip(got, want))
    assert torch.equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):
        ulp = {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}.get(a.dtype, 0.0)
        assert ((a.float() - b.float()).abs() <= ulp * b.float().abs() + 1e-5 * b.float().abs().max()).all()
    for with_native in (True, False):
        ex.impl._native = native if with_native else None
        with pytest.raises(RuntimeError):
            DCPAttention.apply(ex, False, False, lq[:-1], lkv)
    ex.impl._native = native
    ex.impl.time_calls = True        # the phases are looked at: the general path
    assert ex.impl.native() is None


@pytest.mark.parametrize("raw,heads,kv_heads,head_dim,dtype,mask", [([1000, 300, 2100, 640], 8, 2, 128, torch.bfloat16, "causal"),
                                                                    ([1000, 300, 2100, 640], 8, 2, 64, torch.float32, "causal"),
                                                                    ([640, 1100, 900], 16, 4, 96, torch.float16, "shared_question"),
                                                                    ([700], 4, 1, 128, torch.bfloat16, "lambda")])
def test_short_calls_repeat_to_the_bit(raw, heads, kv_heads, head_dim, dtype, mask):
    """Output and gradients of a short batch have the same bits in every call, whatever goes on in between."""
    _need_gpu()
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.runtime.interface import DCPAttention, prepare_dcp_distributed_attn_for_test
    dev = torch.device("cuda", 0)
    ex, lq, lkv, ldo, *_ = prepare_dcp_distributed_attn_for_test(raw, heads, kv_heads, head_dim, 256, heads, get_default_execution_context(1, 1),
                                                                 0, mask, dtype, 3, device=dev, executor_impl="fused")
    lq.requires_grad_(True), lkv.requires_grad_(True)
    first = None
    for i in range(40):
        if i % 3 == 0:
            torch.full((1 << 26,), float("nan"), device=dev)       # other lines in L2, other bytes in what a call allocates
        out = DCPAttention.apply(ex, False, False, lq, lkv)
        got = (out.detach(), *torch.autograd.grad(out, (lq, lkv), ldo))
        if i % 2:
            got[1].cpu()
        first = first or got
        assert all(torch.equal(a, b) for a, b in zip(got, first))
    ex.impl.check_status()


@pytest.mark.parametrize("head_dim,dtype,rise,values", [(64, torch.float32, 54, 90), (64, torch.float16, 70, 0), (96, torch.bfloat16, 54, 90),
                                                        (128, torch.float32, 70, 0), (128, torch.bfloat16, 54, 90)])
def test_rising_scores_in_the_callers_form(head_dim, dtype, rise, values):
    """Scores that rise by 2^rise behind the first key tile, with values of 2^values (a second pass over those tiles of queries), results
    in the caller's type and width: within 2^-6 of the largest value of dense attention, as in the kernel's own tests."""
    _need_gpu()
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.planner import masks
    from dcp_b200.runtime.interface import DCPAttention, prepare_dcp_distributed_attn_for_test
    from dcp_b200.runtime.layout import get_local_q_kv
    from dcp_b200.runtime.simulate import dense_reference
    dev, ctx, raw = torch.device("cuda", 0), get_default_execution_context(1, 1), [700, 260]
    ex, _, _, _, q, kv, _, (wl, _), pad = prepare_dcp_distributed_attn_for_test(raw, 4, 2, head_dim, 256, 4, ctx, 0, "causal", dtype, 5,
                                                                               device=dev, executor_impl="fused")
    scale = head_dim ** -0.5
    q[:, :2, 0] = 16.0
    pos = torch.cat([torch.arange(n) for n in raw])
    kv[:, 0, 0, 0] = ((pos >= 128) * (rise / (16.0 * scale * 1.4427))).to(dtype)
    kv[:, 1] *= 2.0 ** values
    q, kv = q.bfloat16().to(dtype), kv.bfloat16().to(dtype)
    lq, lkv = (t.to(dev) for t in get_local_q_kv(q, kv, wl, ctx.devices()[0], raw))
    out = DCPAttention.apply(ex, False, False, lq, lkv)
    torch.cuda.synchronize()
    ex.impl.check_status()
    ref, *_ = dense_reference(q, kv, raw, pad, masks.get_mask_fn("causal")(raw, pad, torch.int32), scale)
    assert out.dtype == dtype and out.shape == lq.shape
    assert ((out.cpu().double() - ref).abs() <= 2.0 ** -6 * ref.abs().max()).all()


def _executor_with_idle_block(head_dim, dtype, dev):
    """700 + 129 tokens in blocks of 256, causal, but the second block's queries see nothing; and its operands."""
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.planner import masks
    from dcp_b200.planner.compiler import CompilerConfig, InstrCompiler
    from dcp_b200.planner.workload import generate_workload, pad_seqlens
    from dcp_b200.runtime.interface import get_executor
    raw, block, ctx = [700, 129], 256, get_default_execution_context(1, 1)
    padded = pad_seqlens(raw, block)
    mask = masks.get_mask_fn("causal")(raw, padded, torch.int32).clone()
    mask[256:512] = 0
    wl = generate_workload((sum(padded), 4, head_dim), (sum(padded), 2, 2, head_dim), raw, padded, block, 4, ctx.comp_cost_model, mask, dtype)
    fw_wl, bw_wl, fw, bw = InstrCompiler(ctx, CompilerConfig()).compile(wl)
    one = ctx.devices()[0]
    ex = get_executor(4, head_dim, ctx, fw[one], fw_wl, bw[one], bw_wl, executor_impl="fused", device=dev)
    g = torch.Generator().manual_seed(0)
    return (ex, *(torch.randn(829, *heads, head_dim, generator=g).to(dtype).to(dev) for heads in ((4,), (2, 2), (4,))))


@pytest.mark.parametrize("head_dim,dtype", [(128, torch.bfloat16), (64, torch.float32)])
def test_native_calls_leave_idle_rows_zero(head_dim, dtype):
    """Rows of a query block that no tile covers are zero in the output and in dQ, whatever their memory held before, and all else is
    what the general path gives."""
    _need_gpu()
    from dcp_b200.runtime.interface import DCPAttention
    dev = torch.device("cuda", 0)
    ex, q, kv, do = _executor_with_idle_block(head_dim, dtype, dev)
    native = _Recorder(ex.impl.native())
    q.requires_grad_(True), kv.requires_grad_(True)
    res = []
    for ex.impl._native in (native, None):
        junk = [torch.full((829 * 8, head_dim), float("nan"), dtype=dtype, device=dev) for _ in range(8)]
        del junk                                        # the results' memory comes from here
        out = DCPAttention.apply(ex, False, False, q, kv)
        res.append((out.detach(), *torch.autograd.grad(out, (q, kv), do)))
    ex.impl.check_status()
    assert native.taken == [True, True]
    (out, dq, dkv), want = res
    assert not out[256:512].any() and not dq[256:512].any() and out[:256].abs().min() > 0
    assert torch.equal(out, want[0])
    for a, b in zip((dq, dkv), want[1:]):
        assert ((a - b).float().abs() <= 2.0 ** -7 * b.float().abs() + 1e-5 * b.float().abs().max()).all()


@pytest.mark.parametrize("head_dim,dtype", [(128, torch.bfloat16), (64, torch.float32)])
def test_native_calls_on_another_stream_and_in_a_graph(head_dim, dtype):
    """The whole call on a stream of its own, behind work of that stream, and captured and replayed on other inputs: the same
    bits (a short batch)."""
    _need_gpu()
    from dcp_b200.core.common import get_default_execution_context
    from dcp_b200.runtime.interface import DCPAttention, prepare_dcp_distributed_attn_for_test
    dev = torch.device("cuda", 0)
    ex, lq, lkv, ldo, *_ = prepare_dcp_distributed_attn_for_test([300, 129], 4, 2, head_dim, 256, 4, get_default_execution_context(1, 1),
                                                                 0, "causal", dtype, 3, device=dev, executor_impl="fused")
    ex.impl._native = native = _Recorder(ex.impl.native())
    q, kv, do = torch.zeros_like(lq, requires_grad=True), torch.zeros_like(lkv, requires_grad=True), torch.zeros_like(ldo)

    def call():
        out = DCPAttention.apply(ex, False, False, q, kv)
        return (out.detach(), *torch.autograd.grad(out, (q, kv), do))

    def put(*tensors):
        with torch.no_grad():
            for dst, src in zip((q, kv, do), tensors):
                dst.copy_(src)

    first, second = (lq, lkv, ldo), (lq * 0.5, lkv + 1, ldo.flip(0))
    want = []
    for x in (first, second):
        put(*x)
        want.append(call())
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)                   # 10 ms: a launch on another stream would read what was there before
        put(*first)
        got = call()
    side.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want[0]))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = call()
    for x, w in zip((second, first), want[::-1]):
        put(*x)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, w))
    ex.impl.check_status()
    assert all(native.taken)
