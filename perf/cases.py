"""The work that users of this framework have it do on one GPU, as cases that a timing harness can prepare and run.

Four kinds, each through the public entry points that a training or scoring program calls:

* ``train``  one optimizer step of a language model (``lm_trainer.make_train_step`` under ``mpmd_jit_with_loop``):
  microbatch loop, forward, backward, AdamW on fp32 master weights.  Outputs: the losses and the updated state.
* ``encoder`` losses, predictions and gradients of the post-LayerNorm encoder (the example's model).
* ``moe``    forward and backward of a mixture-of-experts feed-forward half-block over microbatches.
* ``score``  the forward pass alone (``mpmd_jit_by_yield``): logits and log-likelihoods of token sequences.

Widths are those of the named configurations (Llama-2-7B / 70B, GPT-2-XL, Mixtral-8x7B) and of the tests and examples;
depth is cut to a few blocks, since every block repeats the same work.
"""
from __future__ import annotations

import functools
import math

import torch
from torch.utils import _pytree as pytree

import jaxpp_b200 as jp
from jaxpp_b200.models import lm_trainer as lt
from jaxpp_b200.models import transformer as tf
from jaxpp_b200.ops import core as ops

DEVICE = "cuda"


def _train(name, family, d, layers, heads, kv, ffn, vocab, seq, n_mb, mb, stages=1, schedule="1f1b", recompute=False, clip=0.0,
           bf16_grads=False):
    return {"name": name, "kind": "train", "family": family, "d": d, "layers": layers, "heads": heads, "kv": kv, "ffn": ffn,
            "vocab": vocab, "seq": seq, "n_mb": n_mb, "mb": mb, "stages": stages, "schedule": schedule, "recompute": recompute,
            "clip": clip, "bf16_grads": bf16_grads}


def listed():
    return [
        # a first run of the framework: the model of the inference example, where launches and host time are everything
        _train("llama_tiny", "llama", 256, 2, 4, 2, 512, 512, 128, 2, 2, stages=2, schedule="interleaved"),
        # a small research model on a few short documents: odd sequence length, gradient clipping
        _train("llama_small", "llama", 1024, 2, 16, 4, 2752, 32000, 1001, 2, 3, clip=1.0),
        # the headline shape: Llama-2-7B blocks, 4096 tokens a microbatch
        _train("llama7b", "llama", 4096, 2, 32, 32, 11008, 32000, 4096, 4, 1),
        # the same blocks fine-tuned on long documents with activation recompute
        _train("llama7b_long", "llama", 4096, 2, 32, 32, 11008, 32000, 16384, 1, 1, recompute=True),
        # Llama-2-70B blocks: grouped-query attention, split backward, recompute, bf16 accumulators
        _train("llama70b", "llama", 8192, 1, 64, 8, 28672, 32000, 4096, 2, 1, schedule="zb", recompute=True, bf16_grads=True),
        # GPT-2-XL blocks as one replica of the data-parallel configuration sees them: one sequence a microbatch
        _train("gpt2xl", "gpt2", 1600, 2, 25, 25, 6400, 50257, 1024, 4, 1),
        # the same blocks with a full GPU's worth of sequences and clipping
        _train("gpt2xl_batch", "gpt2", 1600, 2, 25, 25, 6400, 50257, 1024, 2, 16, clip=1.0),
        # the example encoder of the CPU configuration, in bf16 as the GPU kernels take it
        {"name": "encoder", "kind": "encoder", "d": 256, "layers": 4, "heads": 4, "ffn": 1024, "seq": 128, "n_mb": 4, "mb": 8},
        # a Mixtral-8x7B feed-forward half-block, two sequences a microbatch
        {"name": "mixtral_ffn", "kind": "moe", "d": 4096, "ffn": 14336, "experts": 8, "tokens": 8192, "n_mb": 2},
        # a small mixture of experts with a ragged number of tokens
        {"name": "moe_small", "kind": "moe", "d": 512, "ffn": 1024, "experts": 8, "tokens": 1000, "n_mb": 2},
        # scoring a batch of long documents with Llama-2-7B blocks
        {"name": "score_llama7b", "kind": "score", "d": 4096, "layers": 4, "heads": 32, "kv": 32, "ffn": 11008, "vocab": 32000,
         "seq": 4096, "mb": 2, "stages": 4},
        # scoring one short prompt: a few rows against whole weight matrices
        {"name": "score_short", "kind": "score", "d": 4096, "layers": 4, "heads": 32, "kv": 8, "ffn": 11008, "vocab": 32000,
         "seq": 77, "mb": 1, "stages": 2},
    ]


def _log(rng, lo, hi, step=1):
    return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    """One more case of the ranges above; nothing costs more than the largest listed one."""
    most = max(work(c)["flops"] for c in listed()) * 0.6
    while True:
        kind = rng.choice(["train", "train", "train", "encoder", "moe", "score"])
        hd = rng.choice([64, 128])
        heads = _log(rng, 4, 32)
        kv = rng.choice([k for k in (1, 2, 4, 8, 16, heads) if heads % k == 0])
        d = heads * hd
        seq = rng.choice([_log(rng, 100, 8192), _log(rng, 128, 8192, 64)])
        if kind == "train":
            family = rng.choice(["llama", "llama", "gpt2"])
            schedule = rng.choice(["1f1b", "zb", "interleaved"])
            stages = 2 if schedule == "interleaved" else 1
            c = {"kind": "train", "family": family, "d": d, "layers": 2, "heads": heads, "kv": kv if family == "llama" else heads,
                 "ffn": _log(rng, 2 * d, 4 * d, 8), "vocab": _log(rng, 500, 50000), "seq": seq, "n_mb": rng.randint(1, 4),
                 "mb": rng.randint(1, 6), "stages": stages, "schedule": schedule, "recompute": rng.random() < 0.3,
                 "clip": rng.choice([0.0, 1.0]), "bf16_grads": rng.random() < 0.2}
        elif kind == "encoder":
            c = {"kind": "encoder", "d": d, "layers": 4, "heads": heads, "ffn": _log(rng, 2 * d, 4 * d, 8),
                 "seq": min(seq, 2048), "n_mb": rng.randint(1, 4), "mb": rng.randint(1, 8)}
        elif kind == "moe":
            c = {"kind": "moe", "d": _log(rng, 256, 4096, 64), "ffn": _log(rng, 512, 8192, 64), "experts": rng.choice([4, 8, 16]),
                 "tokens": _log(rng, 200, 12000), "n_mb": rng.randint(1, 3)}
        else:
            c = {"kind": "score", "d": d, "layers": 4, "heads": heads, "kv": kv, "ffn": _log(rng, 2 * d, 4 * d, 8),
                 "vocab": _log(rng, 500, 50000), "seq": _log(rng, 10, 8192), "mb": rng.randint(1, 4), "stages": rng.choice([1, 2, 4])}
        if work(c)["flops"] <= most:
            return c


# ---- what a user's program sets up once: configuration, mesh, compiled step ------------------------------------------
def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _config(case):
    kind = case["kind"]
    if kind == "moe":
        return tf.ModelConfig("mixtral", 32000, case["d"], 1, 32, 8, case["ffn"], case["tokens"], n_experts=case["experts"])
    if kind == "encoder":
        return tf.ModelConfig("encoder", 0, case["d"], case["layers"], case["heads"], case["heads"], case["ffn"], case["seq"],
                              causal=False)
    family = case.get("family", "llama")
    return tf.ModelConfig(family, case["vocab"], case["d"], case["layers"], case["heads"], case["kv"], case["ffn"], case["seq"],
                          n_stages=case["stages"], recompute=case.get("recompute", False))


def _schedule(case):
    name = case.get("schedule", "1f1b")
    return jp.ZeroBubble(1) if name == "zb" else jp.Interleaved1F1B(2, 1) if name == "interleaved" else jp.Std1F1B(1)


def _mesh():
    return jp.MpmdMesh.create({"mpmd": 1, "data": 1, "model": 1}, kind="cuda", multi_process=False)


@functools.lru_cache(maxsize=None)
def _program(key):
    case = dict(key)
    cfg, kind = _config(case), case["kind"]
    schedule = _schedule(case)
    if kind == "train":
        hyper = lt.Hyper(clip_grad_norm=case["clip"] or None, fp32_wgrad=not case["bf16_grads"])
        return jp.mpmd_jit_with_loop(lt.make_train_step(cfg, schedule, hyper), _mesh())
    if kind == "encoder":
        def step(params, batch):
            def microbatch(mb):
                def loss_fn(p):
                    out = tf.encoder_forward(cfg, p, mb)
                    return tf.ops.mse_loss(out, mb) / batch.shape[0], out

                return jp.value_and_grad(loss_fn, has_aux=True)(params)

            return jp.treduce(microbatch, batch, schedule=schedule)

        return jp.mpmd_jit_with_loop(step, _mesh())
    if kind == "moe":
        def step(params, xs, gs):
            def microbatch(mb):
                x, g = mb

                def loss_fn(p, x_):
                    y, aux = tf.mixtral_ffn(cfg, p, x_)
                    return jp.mark_stage_end((y * g).sum().float() + cfg.aux_coef * aux * x_.shape[0])

                prev, ops.WGRAD_DTYPE[0] = ops.WGRAD_DTYPE[0], torch.float32    # fp32 gradients out of the GEMMs
                try:
                    loss, (grads, dx) = jp.value_and_grad(loss_fn, argnums=(0, 1), grad_dtype=torch.float32)(params, x)
                finally:
                    ops.WGRAD_DTYPE[0] = prev
                return (loss, dx), grads

            return jp.treduce(microbatch, (xs, gs), schedule=schedule)

        return jp.mpmd_jit_with_loop(step, _mesh())

    def score(params, tokens, rope):
        inp, nxt = tokens[:, :-1], tokens[:, 1:]
        x = ops.embedding(inp.reshape(-1), params["embed"])
        x = tf.run_layers(cfg, params, x, inp.shape[0], rope)
        x = ops.rmsnorm(x, params["final_norm"], cfg.eps)[0]
        logits = ops.linear(x, params["lm_head"], None)
        nll, _ = ops.cross_entropy(logits, nxt.reshape(-1))
        return jp.mark_stage_end((logits, -nll.view(inp.shape[0], -1).sum(-1)))

    return jp.mpmd_jit_by_yield(score, _mesh())


# ---- what it has in hand before each call ----------------------------------------------------------------------------
def _bias_noise(tree, gen):
    """Biases and norm weights as training leaves them: away from exactly 0 and 1."""
    return pytree.tree_map(lambda p: p + (0.02 * torch.randn(p.shape, generator=gen, device=p.device)).to(p.dtype) if p.dim() == 1 else p,
                           tree)


def prepare(case, seed):
    cfg = _config(case)
    gen = torch.Generator(device=DEVICE).manual_seed(seed * 7 + 1)
    tokens = lambda *shape: torch.randint(0, cfg.vocab, shape, generator=gen, device=DEVICE)
    normal = lambda *shape: torch.randn(*shape, generator=gen, device=DEVICE, dtype=torch.bfloat16)
    state = {"program": _program(_key(case)), "kind": case["kind"]}
    if case["kind"] == "moe":
        layer = _bias_noise(tf.init_layer(cfg, 0, DEVICE, seed), gen)
        params = {k: layer[k] for k in ("ffn_norm", "router", "e_up", "e_down")}
        state["args"] = (params, normal(case["n_mb"], case["tokens"], case["d"]),
                         1e-2 * normal(case["n_mb"], case["tokens"], case["d"]))
        return state
    params = _bias_noise(tf.init_params(cfg, DEVICE, seed), gen)
    if case["kind"] == "encoder":
        state["args"] = (params, normal(case["n_mb"], case["mb"], case["seq"], case["d"]))
    elif case["kind"] == "score":
        state["args"] = (params, tokens(case["mb"], case["seq"] + 1), tf.rope_tables(cfg, DEVICE))
    else:
        # in the middle of training: moments that look like the gradients', a step count past the bias correction
        f32 = lambda fill: pytree.tree_map(fill, params)
        scale = 1e-5
        state["state"] = {
            "params": params, "master": f32(lambda p: p.float()),
            "m": f32(lambda p: torch.randn(p.shape, generator=gen, device=DEVICE).mul_(0.3 * scale)),
            "v": f32(lambda p: torch.rand(p.shape, generator=gen, device=DEVICE).add_(0.5).mul_(scale * scale)),
            "step": torch.full((), 1000, dtype=torch.int64, device=DEVICE)}
        t = tokens(case["n_mb"], case["mb"], case["seq"] + 1)
        state["batch"] = (t[:, :, :-1].contiguous(), t[:, :, 1:].contiguous())
    return state


def run(state):
    if state["kind"] == "train":
        state["state"], losses = state["program"](state["state"], *state["batch"])
        new = state["state"]
        n = len(pytree.tree_leaves(new["params"], is_leaf=lambda x: isinstance(x, jp.MpmdArray)))
        # all of it where it comes to few enough tensors; the compute copy is the master weights rounded, and the second
        # moment comes from the same gradient as the first
        keys = ("params", "master", "m", "v") if 4 * n <= 62 else ("master", "m")
        out = (losses, [new[k] for k in keys])
    else:
        out = state["program"](*state["args"])
    return pytree.tree_map(lambda x: x.local_tensor() if isinstance(x, jp.MpmdArray) else x, out,
                           is_leaf=lambda x: isinstance(x, jp.MpmdArray))


# ---- what one pass cannot do without ---------------------------------------------------------------------------------
def work(case):
    cfg, kind = _config(case), case["kind"]
    d, f = cfg.d_model, cfg.ffn
    if kind == "moe":
        tokens = case["n_mb"] * case["tokens"]
        params = 3 * d * f * case["experts"] + d * case["experts"]
        return {"bytes": params * (2 + 4) + tokens * d * 2 * 3, "flops": 6.0 * tokens * (3 * d * f * cfg.top_k + d * case["experts"])}
    params = cfg.n_params()
    if kind == "encoder":
        tokens = case["n_mb"] * case["mb"] * case["seq"]
        return {"bytes": params * 4 + tokens * d * 4, "flops": cfg.flops_per_token() * tokens}
    if kind == "score":
        tokens = case["mb"] * case["seq"]
        return {"bytes": params * 2 + tokens * (8 + 2 * cfg.padded_vocab), "flops": cfg.flops_per_token() / 3 * tokens}
    tokens = case["n_mb"] * case["mb"] * case["seq"]
    # master, m and v are read and written, the compute copy is read and written
    return {"bytes": params * 28 + tokens * 16, "flops": cfg.flops_per_token() * tokens}


def tolerance(case):
    """Measured between the native kernels and the ATen forms of the same ops (bf16 tensors, fp32 sums in another order),
    worst over all outputs of a case: 1.0e-2 to 1.9e-2 for whole train steps (second moments, which are squares, lead),
    1.5e-2 for the encoder's gradients, 1.6e-2 for logits, 2.1e-2 for expert gradients where a token's second expert is a
    tie; single elements up to 0.31 of the root mean square (0.11 for the encoder and logits)."""
    return {"rel": 0.03, "max": 0.4 if case["kind"] in ("encoder", "score") else 0.99}
