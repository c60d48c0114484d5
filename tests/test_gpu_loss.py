"""Capped-logit cross-entropy kernels (tg_softcap_ce_fwd / _bwd) against the CPU oracle.

Tolerances: per-token nll and lse within 2e-6 relative + 2e-6 absolute of the float64 oracle
(the kernel sums exp() in float32); the bf16 tanh values bit-exact except where float32 tanhf
and float64 tanh round differently (bounded below at 99.9 % equal, never more than one bf16
ulp apart); gradients within rtol 2e-2 / atol 1e-2 * RMS, the bar stated for gradients.
"""
import numpy as np
import pytest
import torch

from oracle import fp8_oracle as fo
from oracle import loss_oracle as lo
from tests.gpu_util import from_torch_bf16, to_torch_bf16

pytestmark = pytest.mark.gpu


def _case(rows, vocab, seed, spread=6.0):
    rng = np.random.default_rng(seed)
    x = (rng.standard_normal((rows, vocab)) * spread).astype(fo.BF16)
    t = rng.integers(0, vocab, size=rows).astype(np.int32)
    return x, t


@pytest.mark.parametrize("rows,vocab,spread", [(7, 512, 6.0), (33, 50304, 3.0), (4, 2056, 40.0),
                                               (5, 50257, 3.0), (3, 12, 2.0), (2, 2049, 6.0)])   # 50257: train-gpt config.py:8
def test_forward_matches_oracle(rows, vocab, spread):
    from train_gpt_b200 import ops
    x, t = _case(rows, vocab, rows + vocab, spread)
    nll, lse, th = ops.softcap_ce_fwd(to_torch_bf16(x), torch.from_numpy(t).cuda(), 15.0)
    z_ref, t_ref = lo.softcap(x, 15.0)
    _, nll_ref, lse_ref = lo.cross_entropy(z_ref, t)
    assert th.shape == (rows, vocab)
    th_bits = from_torch_bf16(th).view(np.uint16).astype(np.int32)
    ref_bits = t_ref.view(np.uint16).astype(np.int32)
    assert np.abs(th_bits - ref_bits).max() <= 1
    assert (th_bits == ref_bits).mean() > 0.999
    assert np.allclose(lse.cpu().numpy(), lse_ref, rtol=2e-6, atol=2e-6)
    assert np.allclose(nll.cpu().numpy(), nll_ref, rtol=2e-5, atol=2e-5)


def test_every_finite_bf16_logit():
    """All 65280 finite bf16 values as logits of one long row: the capped values the kernel
    implies (through lse) and its tanh output follow the oracle over the whole input domain."""
    from train_gpt_b200 import ops
    bits = np.concatenate([np.arange(0, 0x7F80), np.arange(0x8000, 0xFF80)]).astype(np.uint16)
    x = bits.view(fo.BF16).reshape(1, -1)                      # 65280 = 8 * 8160 columns
    t = np.array([12345], dtype=np.int32)
    nll, lse, th = ops.softcap_ce_fwd(to_torch_bf16(x), torch.from_numpy(t).cuda(), 15.0)
    z_ref, t_ref = lo.softcap(x, 15.0)
    _, nll_ref, lse_ref = lo.cross_entropy(z_ref, t)
    d = np.abs(from_torch_bf16(th).view(np.uint16).astype(np.int32) - t_ref.view(np.uint16).astype(np.int32))
    assert d.max() <= 1 and (d == 0).mean() > 0.999
    assert np.allclose(lse.cpu().numpy(), lse_ref, rtol=2e-6) and np.allclose(nll.cpu().numpy(), nll_ref, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("rows,vocab", [(9, 512), (16, 50304), (6, 50257), (5, 12)])
def test_backward_matches_oracle(rows, vocab):
    from train_gpt_b200 import ops
    x, t = _case(rows, vocab, 3 * rows + vocab, 4.0)
    tt = torch.from_numpy(t).cuda()
    _, lse, th = ops.softcap_ce_fwd(to_torch_bf16(x), tt, 15.0)
    gs = torch.tensor([0.75], dtype=torch.float32, device="cuda")
    d = ops.softcap_ce_bwd(th, tt, lse, gs, 15.0)
    th2 = torch.full((rows, th.stride(0)), 7.0, dtype=torch.bfloat16, device="cuda")      # same row pitch, marked padding
    th2[:, :vocab].copy_(th)
    d_inplace = ops.softcap_ce_bwd(th2[:, :vocab], tt, lse, gs, 15.0, in_place=True)
    assert torch.equal(d, d_inplace) and d.shape == (rows, vocab)
    assert bool((th2[:, vocab:] == 7.0).all())                  # nothing is stored past the vocabulary
    ref = lo.softcap_cross_entropy_grad(x, t, 15.0, gscale=0.75)
    got = from_torch_bf16(d).astype(np.float64)
    rms = np.sqrt((ref ** 2).mean())
    assert np.all(np.abs(got - ref) <= 2e-2 * np.abs(ref) + 1e-2 * rms)
    # the target column carries the -1: check it separately, it dominates the row
    assert np.allclose(got[np.arange(rows), t], ref[np.arange(rows), t], rtol=1e-2)


def test_autograd_function_matches_torch_ops():
    """losses.capped_cross_entropy against the op-by-op torch composition of model.py:97 +
    losses.py:9-12 on the same GPU."""
    from train_gpt_b200 import losses
    torch.manual_seed(0)
    logits = (torch.randn(4, 24, 512, device="cuda") * 5).to(torch.bfloat16)
    tg = torch.randint(0, 512, (4, 24), device="cuda")
    a = logits.clone().requires_grad_(True)
    b = logits.clone().requires_grad_(True)
    la = losses.capped_cross_entropy(a, tg, 15.0)
    capped = 15.0 * torch.tanh(b / 15.0)
    lb = torch.nn.functional.cross_entropy(capped.float().view(-1, 512), tg.view(-1))
    (la * 2.0).backward()
    (lb * 2.0).backward()
    assert abs(float(la) - float(lb)) < 2e-5 * abs(float(lb))
    ga, gb = a.grad.float(), b.grad.float()
    rms = gb.pow(2).mean().sqrt()
    assert bool(((ga - gb).abs() <= 2e-2 * gb.abs() + 1e-2 * rms).all())


def test_rejects_bad_arguments():
    from train_gpt_b200 import ops
    with pytest.raises(TypeError):
        ops.softcap_ce_fwd(torch.zeros((2, 16), dtype=torch.bfloat16, device="cuda"),
                           torch.zeros(2, dtype=torch.int64, device="cuda"), 15.0)
    with pytest.raises(ValueError):
        ops.softcap_ce_fwd(torch.zeros((2, 16), dtype=torch.bfloat16, device="cuda"),
                           torch.zeros(2, dtype=torch.int32, device="cuda"), 0.0)          # cap must be positive


def test_reference_default_vocabulary_through_autograd():
    """vocab 50257 (train-gpt config.py:8, not a multiple of 8) through losses.capped_cross_entropy."""
    from train_gpt_b200 import losses
    torch.manual_seed(1)
    logits = (torch.randn(2, 8, 50257, device="cuda") * 4).to(torch.bfloat16)
    tg = torch.randint(0, 50257, (2, 8), device="cuda")
    a = logits.clone().requires_grad_(True)
    b = logits.clone().requires_grad_(True)
    la = losses.capped_cross_entropy(a, tg, 15.0)
    lb = torch.nn.functional.cross_entropy((15.0 * torch.tanh(b / 15.0)).float().view(-1, 50257), tg.view(-1))
    la.backward()
    lb.backward()
    assert abs(float(la) - float(lb)) < 2e-5 * abs(float(lb))
    ga, gb = a.grad.float(), b.grad.float()
    assert ga.shape == gb.shape
    rms = gb.pow(2).mean().sqrt()
    assert bool(((ga - gb).abs() <= 2e-2 * gb.abs() + 1e-2 * rms).all())


@pytest.mark.parametrize("rows,vocab,cap", [(1, 1, 15.0), (3, 7, 15.0), (9, 256, 15.0), (17, 2047, 2.5), (5, 2048, 30.0),
                                            (5, 2049, 15.0), (40, 5119, 15.0), (301, 5121, 64.0), (3, 50257, 15.0), (2, 110000, 15.0),
                                            (2, 130000, 15.0), (4, 300, 80.0)])
def test_one_pass_loss_and_gradient(rows, vocab, cap):
    """The one-pass kernel at the edges of its shapes (one warp or one block per row, rows that start at every alignment,
    ragged last pieces; past its limits in width and cap the two-kernel path), with an upstream gradient of 1 and another."""
    from train_gpt_b200 import losses
    x, t = _case(rows, vocab, rows + vocab, 0.4 * cap)
    x.reshape(-1)[:: 97] = 0
    a = to_torch_bf16(x).requires_grad_(True)
    tt = torch.from_numpy(t.astype(np.int64)).cuda()
    loss = losses.capped_cross_entropy(a, tt, cap)
    loss.backward(retain_graph=True)
    z_ref, _ = lo.softcap(x, cap)
    _, nll_ref, _ = lo.cross_entropy(z_ref, t)
    assert abs(float(loss.detach()) - nll_ref.mean()) <= 1e-5 * abs(nll_ref.mean()) + 1e-6
    for scale in (1.0, 0.75):
        if scale != 1.0:
            a.grad = None
            (loss * scale).backward()
        ref = lo.softcap_cross_entropy_grad(x, t, cap, gscale=scale)
        got = from_torch_bf16(a.grad).astype(np.float64)
        rms = np.sqrt((ref ** 2).mean())
        assert np.all(np.abs(got - ref) <= 2e-2 * np.abs(ref) + 1e-2 * rms)
        assert np.allclose(got[np.arange(rows), t], ref[np.arange(rows), t], rtol=1e-2, atol=1e-12)


def test_one_pass_loss_of_a_nan_row():
    from train_gpt_b200 import losses
    x = torch.zeros(3, 3000, dtype=torch.bfloat16, device="cuda")
    x[1, 1234] = float("nan")
    x.requires_grad_(True)
    loss = losses.capped_cross_entropy(x, torch.zeros(3, dtype=torch.int64, device="cuda"), 15.0)
    loss.backward()
    assert bool(torch.isnan(loss)) and bool(torch.isnan(x.grad[1]).all()) and not bool(torch.isnan(x.grad[::2]).any())


@pytest.mark.parametrize("rows,vocab", [(5, 8), (9, 256), (7, 264), (33, 2048), (6, 2056), (5, 4096), (5, 8904), (3, 50304)])
def test_one_pass_gradient_has_the_bits_of_the_two_kernels(rows, vocab):
    from train_gpt_b200 import losses, ops
    x, t = _case(rows, vocab, rows + vocab, 5.0)
    a, tt = to_torch_bf16(x).requires_grad_(True), torch.from_numpy(t).cuda()
    losses.capped_cross_entropy(a, tt.long(), 15.0).backward()
    _, lse, th = ops.softcap_ce_fwd(a.detach(), tt, 15.0)
    assert torch.equal(a.grad, ops.softcap_ce_bwd(th, tt, lse, None, 15.0))


@pytest.mark.parametrize("rows,vocab", [(1, 256), (2, 8), (3, 40), (31, 8), (100, 64), (127, 16), (128, 256), (130, 8), (255, 8), (511, 24), (1000, 512),
                                        (1024, 256), (2047, 8), (3001, 264), (8192, 2056), (32769, 16), (65536, 8), (70001, 8)])
def test_loss_has_the_bits_of_the_mean_over_tokens(rows, vocab):
    """The loss is the mean that torch takes of the rows' values (which have the bits of the separate forward kernel's)."""
    from train_gpt_b200 import losses, ops
    for seed in range(4):
        x, t = _case(rows, vocab, seed)
        x, t = to_torch_bf16(x), torch.from_numpy(t).cuda()
        want = ops.softcap_ce_fwd(x, t, 15.0)[0].mean()
        assert float(losses.capped_cross_entropy(x, t, 15.0)) == float(want)
        assert float(losses.capped_cross_entropy(x.clone().requires_grad_(), t, 15.0)) == float(want)


# at the edges of the kernel that keeps a row's exponentials in tensor memory: just wide and large enough, one piece more than tensor memory
# holds, the widest, rows that start at every alignment; more rows than the GPU takes at a time, a full last round and a short one.  The last four
# are the other kernel's: a column too narrow and one too wide, rows too few, a last round too short.  Then that kernel where a block's rows start
# at different alignments (three blocks per SM and one: 444 and 148 rows apart).
LARGE_RAGGED = [(2200, 8705, 15.0), (800, 32769, 15.0), (760, 32775, 64.0), (480, 53247, 30.0), (1500, 12301, 0.5), (1200, 20003, 15.0)]
RAGGED = [(2200, 8703, 15.0), (480, 53249, 15.0), (400, 50257, 15.0), (620, 40001, 15.0), (2200, 8193, 15.0), (2220, 8315, 15.0), (1000, 60001, 15.0)]


@pytest.mark.parametrize("rows,vocab,cap", LARGE_RAGGED + RAGGED)
def test_large_ragged_rows(rows, vocab, cap):
    from train_gpt_b200 import losses
    gen = torch.Generator("cuda").manual_seed(rows + vocab)
    x = (torch.randn(rows, vocab, device="cuda", generator=gen) * 0.4 * cap).to(torch.bfloat16)
    t = torch.randint(0, vocab, (rows,), device="cuda", generator=gen)
    t[:8] = torch.tensor([0, 1, 6, 7, vocab - 1, vocab - 2, vocab - 8, 4096])          # in a ragged piece before, after, and in whole ones
    x[3, 5], x[4, 7000], x[5, 9] = float("inf"), float("-inf"), 3e38
    x.requires_grad_(True)
    loss = losses.capped_cross_entropy(x, t, cap)
    with torch.no_grad():
        assert abs(float(losses.capped_cross_entropy(x, t, cap)) - float(loss.detach())) <= 1e-6 * abs(float(loss.detach()))
    loss.backward(retain_graph=True)
    c = torch.tensor(cap, dtype=torch.bfloat16).double()
    bf = lambda v: v.to(torch.bfloat16).double()
    got, total = x.grad, 0.0
    x.grad = None
    (loss * 1e-3).backward()
    for r in range(0, rows, 100):
        th = bf(torch.tanh(bf(x.detach()[r:r + 100].double() / c)))
        z, tt = bf(c * th), t[r:r + 100, None]
        lse = torch.logsumexp(z, -1, keepdim=True)
        total += float((lse - z.gather(1, tt)).sum())
        ref = torch.exp(z - lse).scatter_add_(1, tt, torch.full_like(lse, -1.0)) * (1 - th * th) / rows
        for g, scale in ((got, 1.0), (x.grad, 1e-3)):
            # one bf16 rounding of a float32 value; a tanh at a rounding boundary may fall to its neighbour
            off = (g[r:r + 100].double() - scale * ref).abs() > 2.0 ** -8 * (scale * ref).abs() + 1e-35
            assert float(off.double().mean()) < 1e-4
            assert bool(((g[r:r + 100].double() - scale * ref).abs() <= 2e-2 * (scale * ref).abs() + 1e-2 * scale * ref.square().mean().sqrt()).all())
    assert abs(float(loss.detach()) - total / rows) <= 1e-5 * abs(total / rows)


def test_large_ragged_rows_nan_and_small_scale():
    """A NaN spoils its own row alone; a scale whose product with 1 / sum is no normal number does not lose the gradient."""
    from train_gpt_b200 import losses
    x = torch.randn(2100, 9001, device="cuda").mul(60).to(torch.bfloat16)
    x[7, 1234] = float("nan")
    x.requires_grad_(True)
    t = torch.zeros(2100, dtype=torch.int64, device="cuda")
    loss = losses.capped_cross_entropy(x, t, 64.0)
    loss.backward()
    assert bool(torch.isnan(loss)) and bool(torch.isnan(x.grad[7]).all()) and int(torch.isnan(x.grad).any(1).sum()) == 1
    x = x.detach()[8:].contiguous().requires_grad_(True)
    loss = losses.capped_cross_entropy(x, t[8:], 64.0)
    loss.backward(retain_graph=True)
    base, x.grad = x.grad, None
    (loss * 2.0 ** -40).backward()
    big = base.abs() > 1e-12
    assert bool((x.grad[big] == base[big] * 2.0 ** -40).all())
