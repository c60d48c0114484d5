"""Kernel-level operators: torch CUDA tensors in, torch CUDA tensors out, every one a
single call through the C ABI on torch's current stream.  torch is used for device
memory and streams only; no arithmetic on the path runs in torch.  The argument checks, the
allocation of the outputs and the call itself are native (csrc/host.cpp).

Quantised tensors are `torch.float8_e4m3fn`; scales are float32.
"""
from __future__ import annotations

import torch

from . import _lib
from ._lib import TG_MAJOR_K, TG_MAJOR_MN  # noqa: F401  (what gemm_blockscaled's majors are given as)

F8 = torch.float8_e4m3fn
TILE = 128
_host = _lib.host


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


# ---- quantisers ---------------------------------------------------------------------------

def quantize_rowwise(x: torch.Tensor):
    """1x128 tiles along the last axis (train-gpt fp8.py:39-47 as called at :66).
    x (..., K) bf16 -> q (..., K) e4m3, scales (..., K/128) f32."""
    return _host().quantize_rowwise(x)


def quantize_colwise(x: torch.Tensor):
    """128x1 tiles of a 2-D tensor (what `_quantize_to_fp8(b.T)` at fp8.py:68 computes,
    without the transpose).  x (R, C) bf16 -> q (R, C) e4m3, scales (ceil(R/128), C) f32."""
    return _host().quantize_colwise(x)


def quantize_rowcol(x: torch.Tensor, row_out=None, col_out=None):
    """Row-wise (1x128) and column-wise (128x1) quantisation of a 2-D tensor in one pass.
    Returns (q_row, s_row, q_col, s_col), bit-identical to the two separate kernels.
    `row_out` = (q, s) / `col_out` = (q, s): write that form into these instead of fresh tensors -- column
    slices `big_q[:, c0:c0 + cols]` and `big_s[:, c0 // 128:(c0 + cols) // 128]` (row form) or
    `big_s[:, c0:c0 + cols]` (column form) of wider matrices, unit stride along a row, row pitch a multiple of
    16 bytes: several tensors' forms side by side for one GEMM."""
    if row_out is None and col_out is None:
        return _host().quantize_rowcol(x)
    return _host().quantize_rowcol_into(x, row_out, col_out)


def act_quantize_rowcol(x: torch.Tensor, act: str, gate: torch.Tensor | None = None):
    """quantize_rowcol of an MLP activation computed on the fly from the pre-activation `x`:
    act "relu2" (model.py:72) or "gelu"; "relu2_bwd" / "gelu_bwd" quantise gate * act'(x), the
    gradient at the pre-activation for upstream gradient `gate`.  The activation (or its gradient)
    is rounded to bf16 once and never written to memory.  Returns (q_row, s_row, q_col, s_col)."""
    if act not in _lib.TG_ACT:
        raise ValueError(f"unknown activation {act!r}; use one of {sorted(_lib.TG_ACT)}")
    return _host().act_quantize_rowcol(x, _lib.TG_ACT[act], act, gate)


def quantize_block128(x: torch.Tensor):
    """128x128 tiles.  x (R, C) bf16 -> q (R, C) e4m3, scales (ceil(R/128), C/128) f32."""
    return _host().quantize_block128(x)


def selftest_quantise_division(device="cuda"):
    """Exhaustive check of the quantisers' division shortcut on the device.  Returns
    (pairs checked, mismatches of x*(1/s), of the shipped one-step form, of two steps)."""
    counts = torch.zeros(4, dtype=torch.int64, device=device)
    _lib.check(_lib.load().tg_selftest_quantise_division(_ptr(counts), _stream()), "tg_selftest_quantise_division")
    return tuple(int(v) for v in counts.cpu())


def selftest_bounded_wait(limit_cycles: int = 2_000_000, device="cuda"):
    """Run the GEMM's give-up path (a barrier wait whose clock limit runs out -> abort flag -> every
    role leaves -> tensor memory freed) on a barrier that is never arrived at.  Returns
    (status code, [gave_up == 0, left_early == 2, ordinary_wait_ok == 1, teardown == 1])."""
    status = torch.zeros((1,), dtype=torch.int32, device=device)
    report = torch.zeros((4,), dtype=torch.int32, device=device)
    _lib.check(_lib.load().tg_selftest_bounded_wait(_ptr(status), _ptr(report), int(limit_cycles), _stream()),
               "tg_selftest_bounded_wait")
    return int(status.item()), [int(v) for v in report.cpu()]


# ---- RMSNorm ------------------------------------------------------------------------------

def rmsnorm_fwd(x, gamma, eps: float, pure: bool = False, want_rnorm: bool = False):
    """kernels.py:44-53 (+:66), or kernels.py:30-33 when `pure`.  Returns y [, rnorm]."""
    return _host().rmsnorm_fwd(x, gamma, eps, pure, want_rnorm)


def rmsnorm_quant_fwd(x, gamma, eps: float, pure: bool = False, want_y: bool = False, want_rnorm: bool = False):
    """Norm + 1x128 quantise in one pass.  Returns (q, scales, y or None, rnorm or None)."""
    return _host().rmsnorm_quant_fwd(x, gamma, eps, pure, want_y, want_rnorm)


ADD_NORM_MAX_COLS = 2048     # the widest row the fused add + norm kernels take (one warp holds a row)


def add_rmsnorm_quant_fwd(x, res, gamma, eps: float, pure: bool = False, want_q: bool = True, want_y: bool = True):
    """s = bf16(x + res) (the residual add of model.py:68 / :72), then norm + 1x128 quantise of s, one pass.
    Returns (s, q or None, scales or None, y or None).  Rows wider than ADD_NORM_MAX_COLS: ValueError."""
    return _host().add_rmsnorm_quant_fwd(x, res, gamma, eps, pure, want_q, want_y)


def rmsnorm_bwd(x, gamma, g, eps: float, addend=None):
    """kernels.py:104-118.  Returns (dx bf16 like x, dgamma bf16 (D,)).  With `addend` (bf16 like x, rows of
    at most ADD_NORM_MAX_COLS) dx = bf16(addend + the norm's input gradient): the gradient fan-in of a
    residual junction in the same pass."""
    return _host().rmsnorm_bwd(x, gamma, g, eps, addend)


# ---- capped-logit cross-entropy -----------------------------------------------------------

def softcap_ce_fwd(logits, targets, cap: float, want_tanh: bool = True):
    """model.py:97 + losses.py:9-12 on the uncapped bf16 logits (rows, vocab).
    Returns (nll f32 (rows,), lse f32 (rows,), tanh bf16 (rows, vocab) or None)."""
    return _host().softcap_ce_fwd(logits, targets, cap, want_tanh)


def softcap_ce_bwd(th, targets, lse, gscale, cap: float, in_place: bool = False):
    """Gradient of mean(nll) w.r.t. the uncapped logits; `gscale` is a float32 device scalar
    (or None for 1).  in_place=True overwrites `th` with the gradient."""
    return _host().softcap_ce_bwd(th, targets, lse, gscale, cap, in_place)


# ---- optimiser ------------------------------------------------------------------------------

def sumsq(x, out=None, scratch=None):
    """Sum of squares of a bf16 tensor as a float32 device scalar (one term of optax.global_norm)."""
    return _host().sumsq(x, out, scratch)


def adamw_step(p, g, m, v, step, lr, b1=0.9, b2=0.999, eps=1e-8, weight_decay=0.0, gscale=None):
    """optax clip + adamw on one bf16 parameter tensor, in place (p, m, v).  `step` is an int32
    device scalar holding t (1 for the first step); `gscale` a float32 device scalar or None."""
    _host().adamw_step(p, g, m, v, step, lr, b1, b2, eps, weight_decay, gscale)


# ---- GEMM ---------------------------------------------------------------------------------

def set_gemm_reserved_sms(n: int) -> int:
    """Leave `n` SMs free of the persistent GEMM's thread blocks from the next launch on (for a collective
    that overlaps the GEMMs: the data-parallel gradient all-reduce).  Returns the previous setting."""
    return int(_lib.load().tg_set_gemm_reserved_sms(int(n)))


def new_status(device) -> torch.Tensor:
    """A zeroed device word for the GEMM's bounded-wait status."""
    return torch.zeros((1,), dtype=torch.int32, device=device)


# what the code a GEMM leaves in its status word says about which bounded wait ran out
STATUS_ROLES = {
    1: "the TMA producer waited for a free shared-memory stage",
    2: "the MMA issuer waited for a free accumulator buffer",
    3: "the MMA issuer waited for operands to land",
    4: "the MMA issuer waited for its last instructions to retire",
    5: "the promotion warps waited for an accumulator buffer to fill",
    7: "the store warp waited for a staged tile",
    8: "the promotion warps waited for their staging rows",
    9: "the scale warp waited for a free slot or its block's turn",
}
STATUS_TOKEN = 16   # a training step met a token id outside the vocabulary

def default_status(device) -> torch.Tensor:
    """The status word every gemm_* call on `device` uses when the caller passes none: one word per
    device, allocated once (so a captured CUDA graph keeps pointing at it)."""
    index = torch.device(device).index
    return _host().status_word(-1 if index is None else index)


def status_error(code: int):
    """The exception for a non-zero GEMM status code, or None for 0."""
    if code == 0:
        return None
    if int(code) == STATUS_TOKEN:
        return RuntimeError(f"token id outside the vocabulary (status {int(code)})")
    why = STATUS_ROLES.get(int(code), "unknown role")
    return RuntimeError(f"block-scaled GEMM gave up on a bounded device wait (status {int(code)}: {why}); "
                        "its output is incomplete")


def check_status(status: torch.Tensor | None = None, device=None) -> None:
    """Read a status word (the device's default one if none is given; this synchronises with the
    work queued on it) and raise if a GEMM's bounded wait ran out since it was last zero.  The
    word is cleared so that the next check reports only newer failures."""
    word = status if status is not None else default_status(device if device is not None else "cuda")
    code = int(word.item())
    if code != 0:
        word.zero_()
        raise status_error(code)


def poison_if_failed(value: torch.Tensor, status: torch.Tensor | None = None) -> torch.Tensor:
    """`value` with NaN in place of every element if the status word is non-zero -- a device-side
    select, no synchronisation, capturable in a CUDA graph.  The training step passes its loss through
    this, so a GEMM that gave up surfaces as a NaN loss instead of a silently wrong one."""
    word = status if status is not None else default_status(value.device)
    return torch.where(word.reshape(()) != 0, torch.full_like(value, float("nan")), value)


def gemm_blockscaled(a, b, sa, sb, *, M, N, K, a_major, b_major, sa_strides, sb_strides, sb_gran_n,
                     out_dtype=torch.bfloat16, status=None, out=None, split=True):
    """Raw call of tg_gemm_fp8_blockscaled; see include/train_gpt_b200.h for the argument
    meaning.  a, b are 2-D e4m3 tensors as stored; strides are in elements.  split=True hands
    the library the workspace it asks for (tg_gemm_workspace_bytes), so that a problem with few
    output tiles and a long contraction is cut along the contraction."""
    return _host().gemm(a, b, sa, sb, M, N, K, a_major, b_major, sa_strides, sb_strides, sb_gran_n, out_dtype == torch.float32,
                        status, out, split)


def __getattr__(name):
    if name == "last_gemm_kernel_launches":      # kernels the most recent gemm_* call launched (1, or 2 with a reduce)
        return _host().last_gemm_launches()
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


def _per_column(tile) -> bool:
    return tile == (128, 1) or tuple(tile) == (128, 1)


def gemm_fwd(x_q, x_s, w_q, w_s, weight_tile=(128, 1), out_dtype=torch.bfloat16, status=None):
    """y = x W.  x_q (M,K) rowwise-quantised with x_s (M,K/128); w_q (K,N) with
    w_s (K/128,N) [weight_tile (128,1), from quantize_colwise] or (K/128,N/128)
    [weight_tile (128,128), from quantize_block128]."""
    return _host().gemm_fwd(x_q, x_s, w_q, w_s, _per_column(weight_tile), out_dtype == torch.float32, status)


def gemm_dgrad(g_q, g_s, w_q, w_s, weight_tile=(128, 1), out_dtype=torch.bfloat16, status=None):
    """dx = g W^T (contracts N).  g_q (M,N) rowwise-quantised, g_s (M,N/128); w_q (K,N)
    quantised along N: w_s (K,N/128) [tile (128,1) mode: quantize_rowwise(W)] or the shared
    (K/128,N/128) [tile (128,128)]."""
    return _host().gemm_dgrad(g_q, g_s, w_q, w_s, _per_column(weight_tile), out_dtype == torch.float32, status)


def gemm_wgrad(x_qc, x_sc, g_qc, g_sc, out_dtype=torch.bfloat16, status=None, grad_tile=(128, 1), out=None):
    """dW = x^T g (contracts the tokens).  x_qc (T,K) colwise-quantised (128 tokens x 1),
    scales (ceil(T/128),K).  g_qc (T,N) quantised either the same way, scales (ceil(T/128),N)
    [grad_tile (128,1)], or in 128x128 blocks, scales (ceil(T/128),N/128) [grad_tile (128,128)]:
    one scale per 128 output columns halves the promotion arithmetic and lets the GEMM use its
    128x256 tile.  `out`: a (K, N) bf16 or float32 tensor with unit inner stride to write into (a slice of a
    gradient bucket, say) instead of a new one."""
    return _host().gemm_wgrad(x_qc, x_sc, g_qc, g_sc, _per_column(grad_tile), out_dtype == torch.float32, status, out)
