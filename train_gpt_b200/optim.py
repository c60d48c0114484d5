"""The optimiser of train-gpt's train step on the CUDA path: `make_optimizer(lr, weight_decay,
clip_norm)` (train.py:114-123) = optax.chain(clip_by_global_norm, adamw), for bf16 parameters
whose gradients live in flat buckets (`dp.GradBuckets`).

Global norm: one kernel over all gradient tensors.  Update: one kernel over all parameter tensors --
or over the flat tensors that hold a bucket's parameters, laid out like the bucket's gradients
(`flat=`; optax's adamw has the same hyper-parameters for every leaf, so the update is one
elementwise map over the concatenation) -- that derives the clip factor from the norm and applies
it to the gradient as it reads it, so the clipped gradient is never written.  Norm and step count
stay on the device, which lets the whole step be replayed from a CUDA graph.
"""
from __future__ import annotations

from typing import Sequence

import torch

from . import ops


class ClippedAdamW:
    def __init__(self, params: Sequence[torch.nn.Parameter], lr: float, weight_decay: float = 1e-4, clip_norm: float = 1.0,
                 b1: float = 0.9, b2: float = 0.999, eps: float = 1e-8, flat=None):
        """flat: optional list of (flat parameters, flat gradients, the parameters that are views of the
        former, views) with views(t) = the per-parameter views of a flat tensor t in that layout --
        `dp.GradBuckets.flatten_parameters` / `.views` make them; they must cover `params`."""
        self.params = [p for p in params if p.requires_grad]
        self.lr, self.wd, self.clip, self.b1, self.b2, self.eps = lr, weight_decay, clip_norm, b1, b2, eps
        dev = self.params[0].device
        self._flat = None
        if flat is not None:
            groups = [(fp, fg, list(ps), views) for fp, fg, ps, views in flat if fp.numel()]
            covered = {id(p) for _, _, ps, _ in groups for p in ps}
            if covered != {id(p) for p in self.params}:
                raise ValueError("the flat groups must hold exactly the optimised parameters")
            self._flat, by_id = [], {}
            for fp, fg, ps, views in groups:
                if fp.shape != fg.shape or sum(p.numel() for p in ps) != fp.numel():
                    raise ValueError("flat parameters, flat gradients and their views must have the same length")
                fm, fv = torch.zeros_like(fp), torch.zeros_like(fp)
                self._flat.append((fp, fg, fm, fv))
                for p, m, v in zip(ps, views(fm), views(fv)):
                    by_id[id(p)] = (m, v)
            self.m = [by_id[id(p)][0] for p in self.params]           # per-parameter views of the flat moments
            self.v = [by_id[id(p)][1] for p in self.params]
        else:
            self.m = [torch.zeros_like(p) for p in self.params]           # optax: moments in the parameter dtype
            self.v = [torch.zeros_like(p) for p in self.params]
        self._count = torch.zeros((2,), dtype=torch.int32, device=dev)    # the step count and the update kernel's ticket
        self.step_t = self._count[0]
        self._scratch = (0, None)

    def state_tensors(self):
        return self.m + self.v + [self.step_t]

    def global_norm(self, flat_grads: Sequence[torch.Tensor]) -> torch.Tensor:
        """optax.global_norm (train.py:132) over the flat gradient buckets."""
        flats = [f for f in flat_grads if f.numel()]
        if self._scratch[0] != len(flats):
            self._scratch = (len(flats), ops._host().global_norm_scratch(flats[0], len(flats)))
        return ops._host().global_norm(flats, self._scratch[1])

    def step(self, gnorm: torch.Tensor) -> None:
        """Clip by `gnorm` (optax.clip_by_global_norm: factor clip/norm when norm > clip) and update."""
        if self._flat is not None:
            p, g, m, v = zip(*self._flat)
        else:
            live = [(q.data, q.grad, m, v) for q, m, v in zip(self.params, self.m, self.v) if q.grad is not None]
            p, g, m, v = zip(*live) if live else ((), (), (), ())
        if not p:
            self.step_t += 1
            return
        ops._host().clipped_adamw(p, g, m, v, self._count, gnorm, self.clip, self.lr, self.b1, self.b2, self.eps, self.wd)
