"""Per-block-scaled FP8 matmul: the call surface of train-gpt's `fp8.py` on B200 kernels.

`block_scaled_matmul(a, b, block_k=128)` keeps the reference's signature, error messages
and differentiation contract (train-gpt fp8.py:30-36, :50-78, :85-101): differentiable in
`a` and `b`, `block_k` static, gradients returned in the inputs' dtypes.

Keyword-only extras (defaults reproduce the reference):
  weight_tile  (128, 1)    the reference's weight-scale granularity (it quantises `b.T`
                           along K, fp8.py:68); (128, 128) is the benchmark granularity.
  backward     "bf16_ste"  the reference's straight-through bf16 backward (fp8.py:85-98);
                           "fp8" runs dgrad and wgrad as block-scaled e4m3 GEMMs as well
                           (every operand in 1x128 tiles along its contraction);
                           "fp8_blockgrad" is "fp8" with the upstream gradient quantised in
                           128x128 blocks for wgrad only: coarser, and about twice as fast there.
"""
from __future__ import annotations

import torch

from . import ops

E4M3_MAX = 448.0        # fp8.py:26
DEFAULT_BLOCK_K = 128   # fp8.py:27


def _as_bf16(t: torch.Tensor, name: str) -> torch.Tensor:
    """bf16 view of an operand.  The reference upcasts its bf16 operands to float32 before quantising
    (fp8.py:66,68); these kernels take the bf16 directly.  A wider tensor is taken only if the narrowing
    is exact, so that scales and bytes cannot silently differ from the reference's."""
    if t.dtype == torch.bfloat16:
        return t
    if not t.is_floating_point():
        raise TypeError(f"{name} must be a floating-point tensor, got {t.dtype}")
    n = t.to(torch.bfloat16)
    if not bool((n.to(t.dtype) == t).all()):
        raise TypeError(f"{name} is {t.dtype} with values bf16 cannot hold: the sm_100a kernels quantise bf16 operands "
                        "(as the reference's model does); cast explicitly if that rounding is intended")
    return n


def _quantize_to_fp8(x_f32: torch.Tensor, block_k: int = DEFAULT_BLOCK_K):
    """fp8.py:39-47.  The reference only ever passes an upcast bf16 tensor (fp8.py:66,68), and the
    kernels read bf16: a float32 argument is accepted only if it holds bf16 values exactly (it is then
    narrowed back without loss); anything else raises rather than being rounded silently."""
    K = x_f32.shape[-1]
    if K % block_k != 0:
        raise ValueError(f"K={K} not divisible by block_k={block_k}")
    if block_k != DEFAULT_BLOCK_K:
        raise ValueError(f"block_k={block_k} is not supported by the sm_100a kernels (only {DEFAULT_BLOCK_K})")
    return ops.quantize_rowwise(_as_bf16(x_f32, "x"))


class QuantizedActivation:
    """One activation in the forms the three GEMMs of a linear layer contract: the row-wise
    (1x128) pair for the forward GEMM and, made on first use and then kept, the column-wise
    (128 tokens x 1) pair for wgrad.  Passing the same object as `a_quantized=` to several
    `block_scaled_matmul` calls (q, k, v share one normed activation, model.py:63-65) makes
    each form once instead of once per call, as the reference does (bench_fp8_norm.py:91-93)."""

    def __init__(self, a: torch.Tensor, q=None, scales=None, q_col=None, scales_col=None):
        K = a.shape[-1]
        self.a2d = a.reshape(-1, K)
        self._row = None if q is None else (q.reshape(-1, K), scales.reshape(-1, K // DEFAULT_BLOCK_K))
        self._col = None if q_col is None else (q_col, scales_col)

    @classmethod
    def both(cls, a: torch.Tensor) -> "QuantizedActivation":
        """Both forms from ONE read of `a` (ops.quantize_rowcol): for an activation whose linear layer will be
        differentiated -- the forward GEMM takes the row form now, the weight-gradient GEMM the column form later."""
        K = a.shape[-1]
        a2d = a.reshape(-1, K).to(torch.bfloat16)
        q, s, qc, sc = ops.quantize_rowcol(a2d)
        return cls(a2d, q, s, qc, sc)

    def rowwise(self):
        if self._row is None:
            self._row = ops.quantize_rowwise(self.a2d.to(torch.bfloat16))
        return self._row

    def colwise(self):
        if self._col is None:
            self._col = ops.quantize_colwise(self.a2d.to(torch.bfloat16))
        return self._col


def quantize_weight(b: torch.Tensor, weight_tile=(128, 1)):
    """Quantise b (K, N) for the forward GEMM without transposing it."""
    if tuple(weight_tile) == (128, 1):
        return ops.quantize_colwise(b)
    if tuple(weight_tile) == (128, 128):
        return ops.quantize_block128(b)
    raise ValueError(f"unsupported weight_tile {weight_tile}")


_MODES = {"bf16_ste": 0, "fp8": 1, "fp8_blockgrad": 2}


def _per_column(weight_tile) -> bool:
    tile = tuple(weight_tile)
    if tile not in ((128, 1), (128, 128)):
        raise ValueError(f"unsupported weight_tile {weight_tile}")
    return tile == (128, 1)


def _row_form(a_quantized):
    if a_quantized is None:
        return None, None
    return a_quantized.rowwise() if isinstance(a_quantized, QuantizedActivation) else (a_quantized[0], a_quantized[1])


def _fp8_forward(a, b, block_k=DEFAULT_BLOCK_K, weight_tile=(128, 1), a_quantized=None, return_weight=False):
    """fp8.py:50-78.  `a_quantized` = (q, scales) of `a` made earlier (e.g. by the fused
    norm+quantise kernel) skips the activation quantiser.  return_weight=True also returns the
    quantised weight pair that the GEMM read (128x128 tiles serve the backward's dgrad unchanged; with 128x1
    tiles it has the columns up to the next multiple of 16)."""
    columns, row = _per_column(weight_tile), _row_form(a_quantized)
    n = b.shape[-1]
    if not return_weight or not columns or n % 16 == 0:
        return ops._host().fp8_forward(a, b, block_k, columns, *row, return_weight)
    b = torch.nn.functional.pad(_as_bf16(b, "b"), (0, -n % 16))          # the columns that the pair has and the result has not
    y, weight = ops._host().fp8_forward(a, b, block_k, columns, *row, True)
    y = y[..., :n]
    return (y if y.dim() == 2 else y.contiguous()), weight


def _fp8_backward(block_k, residuals, g, weight_tile=(128, 1), mode="bf16_ste", a_quantized=None, w_quantized=None,
                  b_slot=None):
    """fp8.py:85-98 (mode "bf16_ste"), or the same two GEMMs in block-scaled e4m3.
    `w_quantized`: the forward's 128x128-tile weight pair, reused instead of quantising again.
    `b_slot`: a gradient slot of the weight (see `block_scaled_matmul`); the FP8 modes then write the
    weight gradient there and return None for it."""
    a, b = residuals
    if mode not in _MODES:
        raise ValueError(f"unknown backward mode {mode!r}; use 'bf16_ste', 'fp8' or 'fp8_blockgrad'")
    w_q, w_s = w_quantized if w_quantized is not None else (None, None)
    return ops._host().fp8_backward(a, b, g, _per_column(weight_tile), _MODES[mode],
                                    a_quantized if isinstance(a_quantized, QuantizedActivation) else None, w_q, w_s,
                                    b_slot if b.dtype == torch.bfloat16 else None)


def block_scaled_matmul(a: torch.Tensor, b: torch.Tensor, block_k: int = DEFAULT_BLOCK_K, *,
                        weight_tile=(128, 1), backward: str = "bf16_ste", a_quantized=None) -> torch.Tensor:
    """Per-K-tile block-scaled FP8 matmul.

    a: (..., K), b: (K, N) -> (..., N) bf16.  Requires K % block_k == 0.

    A weight may carry `grad_slot` (an object with take() -> the tensor its gradient belongs in, and
    ready(); train_gpt_b200.dp.GradSlot): in the FP8 backward modes the weight-gradient GEMM then writes
    straight into the flat gradient bucket and autograd gets None, instead of a fresh tensor that is added
    into a zeroed bucket."""
    mode = _MODES.get(backward)
    if mode is None:
        raise ValueError(f"unknown backward mode {backward!r}; use 'bf16_ste', 'fp8' or 'fp8_blockgrad'")
    row_q, row_s = _row_form(a_quantized)
    slot = getattr(b, "grad_slot", None)
    if slot is not None and not (a.dim() >= 2 and b.dim() == 2 and b.shape[1] % 16 == 0 and b.dtype == torch.bfloat16):
        slot = None                              # the direct write takes a bf16 weight as stored, without padding
    return ops._host().block_scaled_matmul(a, b, block_k, _per_column(weight_tile), mode,
                                           a_quantized if isinstance(a_quantized, QuantizedActivation) else None,
                                           row_q, row_s, slot)
