"""What a user of the framework has it compute on one GPU, as measurable cases.

Four kinds of work, all through public entry points:

* ``attention`` - ``get_executor(..., executor_impl="fused")`` with ``DCPAttention.apply``: packed
  variable-length batches, forward only (evaluation) or forward and backward (training);
* ``train``     - ``TrainEngine.train_step``: forward, backward and AdamW of the Llama architecture;
* ``optimizer`` - ``ShardedAdamW.step`` on flat parameter / gradient buffers;
* ``merge``     - ``flash_attn_update_out_lse``: LSE-weighted merge of partial attention results.

Sizes are the ones of the benchmark, the tests and the model configurations of this repository, or
plain multiples of them.
"""
from __future__ import annotations

import dataclasses

import numpy as np
import torch

from dcp_b200.core.common import get_default_execution_context
from dcp_b200.data import synth
from dcp_b200.data.plan_service import plan_batch
from dcp_b200.models.llama import LLAMA3_8B, LlamaModel, tiny_config
from dcp_b200.ops.block_ops import flash_attn_update_out_lse
from dcp_b200.parallel.dist_optimizer import FlatBuffers, ShardedAdamW
from dcp_b200.planner import masks
from dcp_b200.planner.compiler import CompilerConfig, InstrCompiler
from dcp_b200.planner.workload import generate_workload, pad_seqlens
from dcp_b200.runtime.interface import DCPAttention, get_executor
from dcp_b200.train import EngineConfig, TrainEngine

DISTS = {"lognormal8k": synth.LOGNORMAL_8K, "lognormal16k": synth.LOGNORMAL_16K, "mixture": synth.MIXTURE,
         "short": synth.LengthDist("lognormal", 512.0, 0.7, 128, 2048)}
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _attention(name, lens, tokens, lens_seed, heads, kv_heads, mask, block, step, dtype="bf16", head_dim=128, head_block=0):
    """``lens``: explicit lengths ("1000,300,...") or the name of a length distribution that fills
    ``tokens``; ``head_block``: heads per head block (0 = all)."""
    c = {"name": name, "kind": "attention", "lens": lens, "tokens": tokens, "lens_seed": lens_seed, "heads": heads,
         "kv_heads": kv_heads, "head_dim": head_dim, "head_block": head_block or heads, "mask": mask, "block": block,
         "step": step, "dtype": dtype}
    return c


def listed():
    return [
        # a handful of short sequences, few heads: what a unit-sized job or a debug run does; launches and host work count
        _attention("attn_short_causal", "1000,300,2100,640", 4040, 0, 8, 2, "causal", 256, True),
        # fp32 tensors with 64 channels per head (7680 tokens in four sequences): converted and padded on the way in and out
        _attention("attn_fp32_hd64", "512,1024,2048,4096", 7680, 0, 8, 2, "causal", 256, True, "fp32", 64),
        # evaluation: forward only over one packed batch of medium length
        _attention("attn_eval_16k", "lognormal8k", 16384, 0, 32, 8, "causal", 2048, False),
        # one GPU's share of the training benchmark: 32768 tokens of the heavy-tailed length mixture, forward and backward
        _attention("attn_mixture_32k", "mixture", 32768, 1, 32, 8, "causal", 2048, True),
        # structured masks drawn per sequence (sink + window, chunked, shared question), forward and backward
        _attention("attn_masks_32k", "lognormal16k", 32768, 28, 32, 8, "mixed", 2048, True),
        # the attention microbenchmark's whole 131072-token batch, forward and backward: the largest call
        _attention("attn_causal_131k", "lognormal8k", 131072, 0, 32, 8, "causal", 2048, True),
        # a debug-sized model: host work and launches of a whole training step
        {"name": "train_tiny_2k", "kind": "train", "model": "tiny", "hidden": 1024, "layers": 2, "lens": "short",
         "tokens": 2048, "lens_seed": 1, "block": 512},
        # two decoder layers of the 8B width with its vocabulary: every kernel of the training step at its real row sizes
        {"name": "train_8b_width_16k", "kind": "train", "model": "8b", "hidden": 4096, "layers": 2, "lens": "lognormal8k",
         "tokens": 16384, "lens_seed": 2, "block": 2048},
        # optimizer step over the matrices of two decoder layers of the 8B width
        {"name": "optimizer_436m", "kind": "optimizer", "params": 436207616, "buckets": 2, "clip": 1.0},
        # merge of the partial results of four devices for 8192 query tokens
        {"name": "merge_4x8k", "kind": "merge", "partials": 4, "tokens": 8192, "heads": 32},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "attention", "train", "train", "optimizer", "merge"])
    if kind == "merge":
        return {"kind": "merge", "partials": rng.randint(2, 8), "tokens": _log_uniform(rng, 64, 16384),
                "heads": rng.choice([4, 8, 32])}
    if kind == "optimizer":
        return {"kind": "optimizer", "params": 8 * _log_uniform(rng, 1 << 17, 54525952), "buckets": rng.randint(1, 4),
                "clip": rng.choice([0.0, 1.0, 1.0])}
    if kind == "train":
        if rng.random() < 0.6:
            return {"kind": "train", "model": "tiny", "hidden": rng.choice([1024, 2048]), "layers": rng.randint(1, 4),
                    "lens": "short", "tokens": _log_uniform(rng, 512, 8192), "lens_seed": rng.randrange(1 << 20),
                    "block": rng.choice([256, 512])}
        return {"kind": "train", "model": "8b", "hidden": 4096, "layers": rng.randint(1, 2),
                "lens": rng.choice(["lognormal8k", "mixture"]), "tokens": _log_uniform(rng, 2048, 16384),
                "lens_seed": rng.randrange(1 << 20), "block": rng.choice([1024, 2048])}
    most = _pairs(next(c for c in listed() if c["name"] == "attn_causal_131k"))
    while True:
        tokens = _log_uniform(rng, 600, 131072)
        heads, kv_heads = rng.choice([(8, 2), (32, 8), (32, 8), (16, 4), (4, 4)])
        c = _attention("", rng.choice(["lognormal8k", "lognormal16k", "mixture", "short"]), tokens, rng.randrange(1 << 20),
                       heads, kv_heads, rng.choice(["causal", "causal", "lambda", "shared_question", "chunked_first_chunk", "mixed"]),
                       rng.choice([256, 512]) if tokens < 16384 else rng.choice([1024, 2048]), rng.random() < 0.75)
        del c["name"]
        if tokens <= 32768:
            c["dtype"] = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
            c["head_dim"] = rng.choice([128, 128, 128, 64, 96])
            c["head_block"] = rng.choice([heads, heads, heads, heads // 2 if heads // 2 >= kv_heads else heads])
        if _pairs(c) * heads <= most * 32:
            return c


# ---------------------------------------------------------------------------------------- sizes of a case
def _lengths(case):
    if case["lens"] in DISTS:
        return [int(x) for x in synth.sample_seqlens(case["tokens"], DISTS[case["lens"]], case["lens_seed"])]
    return [int(x) for x in case["lens"].split(",")]


def _mask(case, raw, padded):
    mask = case.get("mask", "causal")
    info = synth.assign_mask_kinds(raw, case["lens_seed"]) if mask == "mixed" else None
    return masks.get_mask_fn(mask)(raw, padded, torch.int32, info)


def _pairs(case):
    """(query, key) pairs of one head."""
    raw = _lengths(case)
    if case.get("mask", "causal") == "causal":
        return float(sum(n * (n + 1) // 2 for n in raw))
    m = masks.to_two_range(_mask(case, raw, raw))
    return float(np.maximum(m[:, :, 1] - m[:, :, 0], 0).sum())


def _model(case):
    if case["model"] == "8b":
        return dataclasses.replace(LLAMA3_8B, n_layers=case["layers"])
    h = case["hidden"]
    return tiny_config(n_layers=case["layers"], hidden=h, n_heads=h // 128, n_kv_heads=h // 512, ffn=2 * h, vocab=4096)


# ---------------------------------------------------------------------------------------- state
def _prepare_attention(case, gen, dev):
    H, G, d, bs = case["heads"], case["kv_heads"], case["head_dim"], case["block"]
    dtype = DTYPES[case["dtype"]]
    raw = _lengths(case)
    padded = pad_seqlens(raw, bs)
    ctx = get_default_execution_context(1, 1)
    wl = generate_workload((sum(padded), H, d), (sum(padded), 2, G, d), raw, padded, bs, case["head_block"],
                           ctx.comp_cost_model, _mask(case, raw, padded), dtype)
    fw_wl, bw_wl, fw, bw = InstrCompiler(ctx, CompilerConfig()).compile(wl)
    one = ctx.devices()[0]
    ex = get_executor(case["head_block"], d, ctx, fw[one], fw_wl, bw[one], bw_wl, executor_impl="fused", device=dev)
    p = ex.program
    new = lambda *shape: torch.randn(*shape, generator=gen, device=dev, dtype=torch.float32).to(dtype)
    q, kv = new(p.q_local_rows, p.heads_q, d), new(p.kv_local_rows, 2, p.heads_kv, d)
    state = {"kind": "attention", "ex": ex, "q": q, "kv": kv, "do": None}
    if case["step"]:
        q.requires_grad_(True)
        kv.requires_grad_(True)
        state["do"] = new(p.q_local_rows, p.heads_q, d)
    return state


def _prepare_train(case, seed, dev):
    raw = _lengths(case)
    # the learning rate of an early warm-up step; nothing but layer inputs and attention results is kept for
    # the backward, as with the full model on one GPU
    cfg = EngineConfig(_model(case), tokens_per_step=case["tokens"], block_size=case["block"], lr=1e-6, seed=seed,
                       length_dist=DISTS[case["lens"]], planner_workers=0, activation_budget_gb=0.0)
    eng = TrainEngine(cfg, dev)
    plan = plan_batch(eng.spec, 0, 0, raw, synth.make_token_batch(raw, eng.model.cfg.vocab, seed))
    return {"kind": "train", "eng": eng, "plan": plan}


def _prepare_optimizer(case, gen, dev):
    n, k = case["params"], case["buckets"]
    bufs = FlatBuffers(n, dev)
    bufs.params.normal_(0.0, 0.02, generator=gen)
    bufs.grads.normal_(0.0, 1e-3, generator=gen)
    per = n // k // 8 * 8
    cuts = [(i * per, per if i + 1 < k else n - i * per) for i in range(k)]
    opt = ShardedAdamW(bufs, lr=1e-4, clip_grad=case["clip"] or None, buckets=cuts)
    return {"kind": "optimizer", "opt": opt, "bufs": bufs}


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    if case["kind"] == "attention":
        return _prepare_attention(case, gen, dev)
    if case["kind"] == "train":
        return _prepare_train(case, int(seed) % (1 << 20), dev)
    if case["kind"] == "optimizer":
        return _prepare_optimizer(case, gen, dev)
    n, t, h = case["partials"], case["tokens"], case["heads"]
    return {"kind": "merge",
            "outs": torch.randn(n, t, h, 128, generator=gen, device=dev, dtype=torch.bfloat16),
            "lses": 4.0 + 2.0 * torch.randn(n, t, h, generator=gen, device=dev, dtype=torch.float32)}


# ---------------------------------------------------------------------------------------- one pass
def run(state):
    if state["kind"] == "attention":
        q, kv = state["q"], state["kv"]
        if state["do"] is None:
            with torch.no_grad():
                return DCPAttention.apply(state["ex"], False, False, q, kv)
        out = DCPAttention.apply(state["ex"], False, False, q, kv)
        dq, dkv = torch.autograd.grad(out, (q, kv), state["do"])
        return {"out": out.detach(), "dq": dq, "dkv": dkv}
    if state["kind"] == "train":
        eng = state["eng"]
        loss = eng.train_step(state["plan"])
        o = eng.optimizer
        return {"loss": loss, "grads": eng.bufs.grads, "params": eng.bufs.params, "master": o.master, "m": o.m, "v": o.v}
    if state["kind"] == "optimizer":
        o = state["opt"]
        o.step(1.0)
        return {"params": state["bufs"].params, "master": o.master, "m": o.m, "v": o.v}
    return flash_attn_update_out_lse(state["outs"], state["lses"])


# ---------------------------------------------------------------------------------------- the same in 64 bits
def _exact_attention(case, gen, dev):
    H, G, d, dtype = case["heads"], case["kv_heads"], case["head_dim"], DTYPES[case["dtype"]]
    raw = _lengths(case)
    T, blocks = sum(raw), H // case["head_block"]          # rows: head block by head block, in each all tokens
    hb, gb = H // blocks, G // blocks
    new = lambda *shape: torch.randn(*shape, generator=gen, device=dev, dtype=torch.float32).to(dtype)
    q, kv = new(blocks * T, hb, d), new(blocks * T, 2, gb, d)
    do = new(blocks * T, hb, d) if case["step"] else None
    mask = torch.from_numpy(masks.to_two_range(_mask(case, raw, raw))).to(dev)        # [T, range, bound]
    wide = lambda t: torch.zeros(t.shape, dtype=torch.float64, device=dev)
    out, dq, dkv = wide(q), None if do is None else wide(q), None if do is None else wide(kv)
    step = 4096
    for b in range(blocks):
        lo = 0
        for n in raw:
            own = slice(b * T + lo, b * T + lo + n)
            pos = torch.arange(n, device=dev)
            for h in range(hb):
                g = h * gb // hb
                k, v = kv[own, 0, g].double(), kv[own, 1, g].double()
                for t in range(0, n, step):
                    m = min(step, n - t)
                    rows = slice(own.start + t, own.start + t + m)
                    r = mask[lo + t:lo + t + m]
                    sees = ((pos >= r[:, 0, 0, None]) & (pos < r[:, 0, 1, None])) | ((pos >= r[:, 1, 0, None]) & (pos < r[:, 1, 1, None]))
                    qt = q[rows, h].double()
                    p = ((qt @ k.t()) * d ** -0.5).masked_fill_(~sees, float("-inf")).softmax(1).nan_to_num_(0.0)
                    o = p @ v
                    out[rows, h] = o
                    if do is not None:
                        dot = do[rows, h].double()
                        dkv[own, 1, g] += p.t() @ dot
                        ds = (dot @ v.t()).sub_((o * dot).sum(1, keepdim=True)).mul_(p).mul_(d ** -0.5)
                        dq[rows, h] = ds @ k
                        dkv[own, 0, g] += ds.t() @ qt
            lo += n
    return out if do is None else {"out": out, "dq": dq, "dkv": dkv}


def _exact_optimizer(case, gen, dev):
    n = case["params"]
    p = torch.empty(n, dtype=torch.bfloat16, device=dev).normal_(0.0, 0.02, generator=gen).double()
    g = torch.empty(n, dtype=torch.bfloat16, device=dev).normal_(0.0, 1e-3, generator=gen).double()
    if case["clip"]:
        g *= min(1.0, case["clip"] / (float(g.norm()) + 1e-6))
    # first step of AdamW with betas 0.9 / 0.95, eps 1e-8, weight decay 0.1: the corrected moments are g and g^2
    m, v = 0.1 * g, 0.05 * g * g
    p -= 1e-4 * (g / (g.abs() + 1e-8) + 0.1 * p)
    return {"params": None, "master": p, "m": m, "v": v}


def exact(case, seed):
    """What ``run`` gives on a fresh state, in 64 bits.  A training step has none here: its layers are bf16
    throughout, and its kernels are in the other cases."""
    if case["kind"] == "train":
        return None
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    if case["kind"] == "attention":
        return _exact_attention(case, gen, dev)
    if case["kind"] == "optimizer":
        return _exact_optimizer(case, gen, dev)
    n, t, h = case["partials"], case["tokens"], case["heads"]
    outs = torch.randn(n, t, h, 128, generator=gen, device=dev, dtype=torch.bfloat16).double()
    lses = (4.0 + 2.0 * torch.randn(n, t, h, generator=gen, device=dev, dtype=torch.float32)).double()
    lse = torch.logsumexp(lses, 0)
    return ((lses - lse).exp()[..., None] * outs).sum(0), lse


# ---------------------------------------------------------------------------------------- what a pass needs
def work(case):
    if case["kind"] == "attention":
        H, G, d, t = case["heads"], case["kv_heads"], case["head_dim"], sum(_lengths(case))
        pairs = _pairs(case) * H * d
        size = 4 if case["dtype"] == "fp32" else 2
        rows = t * d * size
        # forward: q, k, v in, out written; backward: also dout in, dq, dk, dv written; two products per pair
        # forward, five backward
        if case["step"]:
            return {"bytes": rows * (4 * H + 4 * G), "flops": 14.0 * pairs}
        return {"bytes": rows * (2 * H + 2 * G), "flops": 4.0 * pairs}
    if case["kind"] == "train":
        m, t = _model(case), case["tokens"]
        n = LlamaModel.flat_size(m)
        dense = m.n_params() - m.vocab * m.hidden       # every parameter but the embedding is multiplied with every token
        # fp32 master weights and moments are read and written, bf16 parameters read and written, gradients written
        return {"bytes": 30.0 * n, "flops": 6.0 * dense * t + 14.0 * _pairs(case) * m.n_heads * m.head_dim * m.n_layers}
    if case["kind"] == "optimizer":
        # gradients in, fp32 master weights and moments in and out, bf16 parameters out
        return {"bytes": 28.0 * case["params"], "flops": 15.0 * case["params"]}
    n, t, h = case["partials"], case["tokens"], case["heads"]
    return {"bytes": float(t * h * (n + 1) * (128 * 2 + 4)), "flops": 2.0 * n * t * h * 128}


def tolerance(case):
    """About four times what a pass differs from its computation in 64 bits (attention, optimizer, merge), or
    from another order of the same bf16 operations (training step), on the listed sizes."""
    if case["kind"] == "attention":
        # bf16 operands, probabilities and score gradients: out 3.4e-3, dq 3.0e-3, dk / dv 2.6e-3 against fp64
        # (4.4e-3 with fp32 tensors, whose conversion to bf16 counts too); single elements up to 0.35 of the rms
        return {"rel": 1.6e-2, "max": 0.9}
    if case["kind"] == "train":
        # bf16 activations and gradients: 1.0e-2 between two passes that only differ in the order of fp32 sums
        return {"rel": 3e-2, "max": 0.9}
    if case["kind"] == "optimizer":
        # fp32 state: 1.0e-6 (second moment); a bf16 parameter may round to its neighbour
        return {"rel": 1e-5, "max": 1e-2}
    # bf16 result of an fp32 merge: 1.7e-3
    return {"rel": 7e-3, "max": 2e-2}
