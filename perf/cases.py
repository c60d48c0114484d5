"""What this library is used for, as cases that can be timed and compared.

A case is a dict of plain values; its "kind" says which of the library's paths it takes:

  serve   a pre-norm linear at inference: `kernels.rms_norm_quant`, then the GEMM against a weight that was
          quantised once when the model was loaded (`fp8.quantize_weight`, `ops.gemm_fwd`)
  linear  one linear in training: `fp8.block_scaled_matmul` forward and backward through autograd
  layer   the four linears of a decoder layer, each forward and backward, the same way
  norm    a normalisation in training, forward and backward: either the fused norm + quantise in front of an
          FP8 linear (`kernels.rms_norm_quant` and `ops.rmsnorm_bwd`) or `kernels.rms_norm` through autograd
  loss    `losses.capped_cross_entropy` forward and backward on the unembedding's output
  train   one optimiser step of `step.Trainer`: loss, backward, clip and AdamW

`prepare` makes what a program holds before the call (inputs, weights, a trainer) and `run` makes one pass.
"""
from __future__ import annotations

import math

import torch

from train_gpt_b200 import fp8, kernels, losses, ops, step

EPS = 1e-6
TILES = {"128x128": (128, 128), "128x1": (128, 1)}


# ---- the cases -------------------------------------------------------------------------------------------------

def listed():
    return [
        # one token of one sequence against a 2048-wide model's q/k/v weight: the smallest call, all latency
        dict(name="serve_1x2048x6144", kind="serve", tokens=1, k=2048, n=6144, tile="128x128"),
        # a decode batch against a wide square weight: one pass over the weight
        dict(name="serve_16x8192x8192", kind="serve", tokens=16, k=8192, n=8192, tile="128x128"),
        # a short prompt, ragged, with the weight scaled per column as the reference does it
        dict(name="serve_200x2048x8192_col", kind="serve", tokens=200, k=2048, n=8192, tile="128x1"),
        # the up projection of the small model in train-gpt's configuration: a training call that is all launches
        dict(name="linear_128x128x512", kind="linear", tokens=128, k=128, n=512, tile="128x128", backward="fp8"),
        # one linear at the size of the single-layer benchmark configuration
        dict(name="linear_4096x768x3072", kind="linear", tokens=4096, k=768, n=3072, tile="128x128", backward="fp8"),
        # the call with its default options (column scales, straight-through bf16 backward), a ragged token count
        dict(name="linear_5000x1024x4096_ste", kind="linear", tokens=5000, k=1024, n=4096, tile="128x1",
             backward="bf16_ste"),
        # the decoder-layer benchmark configuration, full size: the largest FP8 work
        dict(name="layer_32768x2048", kind="layer", tokens=32768, d=2048),
        # the norm benchmark configuration: fused with the quantiser, and its backward
        dict(name="norm_32768x2048_quant", kind="norm", rows=32768, cols=2048, quant=True),
        # a plain norm of wide rows, an odd number of them
        dict(name="norm_3001x4096", kind="norm", rows=3001, cols=4096, quant=False),
        # eight sequences of 1024 tokens against the reference's default vocabulary, which is no multiple of 8
        dict(name="loss_8192x50257", kind="loss", rows=8192, vocab=50257, cap=15.0),
        # a step of train-gpt's small model, launched operation by operation
        dict(name="train_small", kind="train", layers=2, d=128, heads=4, ff=512, vocab=256, seq=128, batch=8,
             act="relu2", graph=False),
        # a step of the pre-training configuration (24 layers, d_model 1024), eight sequences, replayed as a graph
        dict(name="train_24x1024", kind="train", layers=24, d=1024, heads=16, ff=4096, vocab=50304, seq=1024, batch=8,
             act="gelu", graph=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tiles(rng, lo, hi):
    """A multiple of 128, spread over the logarithm."""
    return min(hi, max(lo, 128 * round(_log(rng, lo, hi) / 128)))


def draw(rng):
    kind = rng.choice(("serve", "serve", "linear", "linear", "layer", "norm", "norm", "loss", "train"))
    if kind == "serve":
        return dict(kind=kind, tokens=_log(rng, 1, 256), k=_tiles(rng, 512, 8192), n=_tiles(rng, 512, 8192),
                    tile=rng.choice(("128x128", "128x128", "128x1")))
    if kind == "linear":
        tile, backward = rng.choice((("128x128", "fp8"), ("128x128", "fp8"), ("128x1", "bf16_ste"), ("128x1", "bf16_ste"),
                                     ("128x1", "fp8"), ("128x128", "fp8_blockgrad")))
        k, n = _tiles(rng, 128, 8192), _tiles(rng, 128, 8192)
        if backward == "bf16_ste" and rng.random() < 0.5:
            n += rng.randrange(-100, 101)           # the straight-through mode takes any width
        return dict(kind=kind, tokens=min(_log(rng, 64, 32768), int(1.6e12 / (k * n))), k=k, n=n, tile=tile, backward=backward)
    if kind == "layer":
        return dict(kind=kind, tokens=_log(rng, 1024, 32768), d=_tiles(rng, 512, 2048))
    if kind == "norm":
        quant = rng.random() < 0.5
        cols = _tiles(rng, 128, 8192) if quant else 8 * _log(rng, 16, 1024)
        return dict(kind=kind, rows=min(_log(rng, 64, 32768), int(1.4e8 / cols)), cols=cols, quant=quant)
    if kind == "loss":
        return dict(kind=kind, rows=_log(rng, 128, 8192), vocab=_log(rng, 256, 50304), cap=rng.choice((15.0, 30.0)))
    d = rng.choice((128, 256, 384, 512, 768))
    return dict(kind=kind, layers=rng.randrange(1, 7), d=d, heads=d // 64 if d > 128 else 4, ff=4 * d,
                vocab=8 * _log(rng, 32, 2048), seq=128 * rng.randrange(1, 9), batch=rng.randrange(1, 9),
                act=rng.choice(("gelu", "relu2")), graph=rng.random() < 0.5)


def _layer_shapes(d):
    """(K, N) of q/k/v as one, the attention output, the up and the down projection."""
    return [(d, 3 * d), (d, d), (d, 4 * d), (4 * d, d)]


# ---- inputs ----------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, shape, std=1.0):
    return (torch.randn(shape, device="cuda", generator=gen) * std).to(torch.bfloat16)


def _activations(gen, shape):
    """N(0, 1) with one value in a thousand fifty times as large, as outlier features are."""
    x = torch.randn(shape, device="cuda", generator=gen)
    return torch.where(torch.rand(shape, device="cuda", generator=gen) < 1e-3, 50 * x, x).to(torch.bfloat16)


def _heavy_tailed(gen, shape):
    """Student's t with three degrees of freedom."""
    z = torch.randn((4, *shape), device="cuda", generator=gen)
    return (z[0] / (z[1:].square().mean(0)).sqrt()).to(torch.bfloat16)


def _linear_state(gen, tokens, k, n, tile, backward):
    return {"x": _normal(gen, (tokens, k)).requires_grad_(), "w": _normal(gen, (k, n), 0.02).requires_grad_(),
            "g": _normal(gen, (tokens, n)), "tile": TILES[tile], "backward": backward}


def _bucket_storages(params):
    """The parameters as the flat tensors they are stored in (a trainer keeps several in one)."""
    seen = {}
    for p in params:
        s = p.untyped_storage()
        seen.setdefault(s.data_ptr(), torch.empty(0, dtype=p.dtype, device=p.device).set_(s, 0, (s.nbytes() // p.element_size(),)))
    return list(seen.values())


def prepare(case, seed):
    gen, kind = _gen(seed), case["kind"]
    if kind == "serve":
        tile = TILES[case["tile"]]
        w_q, w_s = fp8.quantize_weight(_normal(gen, (case["k"], case["n"]), 0.02), tile)
        return {"kind": kind, "x": _heavy_tailed(gen, (case["tokens"], case["k"])), "gamma": 1 + _normal(gen, (case["k"],), 0.1),
                "w_q": w_q, "w_s": w_s, "tile": tile}
    if kind == "linear":
        return {"kind": kind, **_linear_state(gen, case["tokens"], case["k"], case["n"], case["tile"], case["backward"])}
    if kind == "layer":
        return {"kind": kind, "linears": [_linear_state(gen, case["tokens"], k, n, "128x128", "fp8")
                                          for k, n in _layer_shapes(case["d"])]}
    if kind == "norm":
        shape = (case["rows"], case["cols"])
        return {"kind": kind, "quant": case["quant"], "x": _activations(gen, shape).requires_grad_(not case["quant"]),
                "gamma": (1 + _normal(gen, (case["cols"],), 0.1)).requires_grad_(not case["quant"]), "g": _normal(gen, shape)}
    if kind == "loss":
        return {"kind": kind, "logits": _normal(gen, (case["rows"], case["vocab"]), 4.0).requires_grad_(), "cap": case["cap"],
                "targets": torch.randint(0, case["vocab"], (case["rows"],), device="cuda", generator=gen)}
    cfg = step.StepConfig(vocab_size=case["vocab"], seq_len=case["seq"], d_model=case["d"], n_layers=case["layers"],
                          n_heads=case["heads"], head_dim=case["d"] // case["heads"], d_ff=case["ff"], activation=case["act"])
    trainer = step.Trainer(cfg, torch.device("cuda", 0), seed=seed, graph=case["graph"])
    ids, targets = step.synthetic_batch(cfg, case["batch"], torch.device("cuda", 0), seed)
    return {"kind": kind, "trainer": trainer, "ids": ids, "targets": targets,
            "parameters": _bucket_storages(trainer.model.parameters())}


# ---- one pass --------------------------------------------------------------------------------------------------

def _run_linear(s):
    s["x"].grad = s["w"].grad = None
    y = fp8.block_scaled_matmul(s["x"], s["w"], weight_tile=s["tile"], backward=s["backward"])
    y.backward(s["g"])
    return {"y": y.detach(), "dx": s["x"].grad, "dw": s["w"].grad}


def run(state):
    kind = state["kind"]
    if kind == "serve":
        h = kernels.rms_norm_quant(state["x"], state["gamma"], EPS)
        return ops.gemm_fwd(h.q, h.scales, state["w_q"], state["w_s"], state["tile"])
    if kind == "linear":
        return _run_linear(state)
    if kind == "layer":
        return [_run_linear(s) for s in state["linears"]]
    if kind == "norm":
        x, gamma, g = state["x"], state["gamma"], state["g"]
        if state["quant"]:
            h = kernels.rms_norm_quant(x, gamma, EPS)
            dx, dgamma = ops.rmsnorm_bwd(x, gamma, g, EPS)
            return {"q": h.q, "scales": h.scales, "dx": dx, "dgamma": dgamma}
        x.grad = gamma.grad = None
        y = kernels.rms_norm(x, gamma, EPS)
        y.backward(g)
        return {"y": y.detach(), "dx": x.grad, "dgamma": gamma.grad}
    if kind == "loss":
        state["logits"].grad = None
        loss = losses.capped_cross_entropy(state["logits"], state["targets"], state["cap"])
        loss.backward()
        return {"loss": loss.detach(), "dlogits": state["logits"].grad}
    trainer = state["trainer"]
    loss, norm = trainer.step(state["ids"], state["targets"])
    # the step's results; the gradients are intermediate here, and the attention library's backward pass (atomic adds)
    # makes those of the first layers differ by 3 % between two runs of the same step
    return {"loss": loss, "norm": norm, "parameters": state["parameters"]}


# ---- what a pass cannot do without, and how close another implementation comes -----------------------------------

def _linear_work(tokens, k, n):
    # x, w, g in; y, dx, dw out
    return 2.0 * (2 * tokens * k + 2 * k * n + 2 * tokens * n), 6.0 * tokens * k * n


def work(case):
    kind = case["kind"]
    if kind == "serve":
        m, k, n = case["tokens"], case["k"], case["n"]
        scales = 4 * (k // 128) * (n // 128 if case["tile"] == "128x128" else n)
        return {"bytes": 2.0 * m * k + 2 * k + k * n + scales + 2 * m * n, "flops": 2.0 * m * k * n}
    if kind == "linear":
        b, f = _linear_work(case["tokens"], case["k"], case["n"])
        return {"bytes": b, "flops": f}
    if kind == "layer":
        each = [_linear_work(case["tokens"], k, n) for k, n in _layer_shapes(case["d"])]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    if kind == "norm":
        e = case["rows"] * case["cols"]
        # x, g and gamma in; the norm's output (bytes and scales, or bf16), dx and dgamma out
        return {"bytes": (2 + 2 + (1 + 4 / 128 if case["quant"] else 2) + 2) * e + 4.0 * case["cols"], "flops": 20.0 * e}
    if kind == "loss":
        e = case["rows"] * case["vocab"]
        return {"bytes": 4.0 * e + 8 * case["rows"], "flops": 20.0 * e}
    tokens, d, ff = case["batch"] * case["seq"], case["d"], case["ff"]
    matrices = case["layers"] * (4 * d * d + 2 * d * ff)
    params = matrices + 2 * case["vocab"] * d + case["seq"] * d
    attention = case["layers"] * 2.0 * tokens * case["seq"] * d             # causal: half of 4 T d per token
    # parameters, gradients and both moments read, all but the gradients written; the residual stream of each layer
    return {"bytes": 16.0 * params + 8.0 * case["layers"] * tokens * d,
            "flops": 6.0 * tokens * (matrices + case["vocab"] * d) + 3.5 * attention}


def tolerance(case):
    if case["kind"] == "train":
        # e4m3 roundings flip where an activation moves by a bf16 ulp, through every layer of the step; a step moves
        # the parameters by 1.4e-2 of their norm, and two runs of one step are 3e-3 apart
        return {"rel": 8e-3}
    if case["kind"] == "norm":
        # one bf16 rounding of dx; an e4m3 byte moves where the sum of squares is added in another order
        return {"rel": 5e-3}
    return {"rel": 1e-2 if case["kind"] != "loss" else 5e-3}       # bf16 results of float32 sums
