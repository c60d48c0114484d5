"""Parity of the CUDA RMSNorm kernels (forward, fused forward+quantise, backward) with the
CPU oracle.

Tolerances.  The row variance is a float32 reduction whose order differs between any two
implementations, so `rnorm` may differ from the oracle's in the last bits; the tests
therefore (a) bound |rnorm - oracle| by 2 ulp and (b) demand BIT-EXACT outputs against the
oracle evaluated with the kernel's own rnorm.  The backward's two row/column sums are
float32 reductions too: dx may differ by one bf16 ulp on a small fraction of elements
(bound: 1 ulp + 2^-14 RMS for cancelled values, < 1 % of elements), dgamma by 2^-7 relative (one bf16 ulp) of its RMS.
"""
import numpy as np
import pytest
import torch

from oracle import fp8_oracle as fo
from oracle import norm_oracle as no
from tests.gpu_util import BF16, f8_bytes, from_torch_bf16, normal_bf16, to_torch_bf16

pytestmark = pytest.mark.gpu


def _ulp_diff_f32(a, b):
    return np.abs(a.view(np.int32).astype(np.int64) - b.view(np.int32).astype(np.int64))


def _inputs(shape, seed, eps):
    rng = np.random.default_rng(seed)
    x = normal_bf16(rng, shape, outlier_p=1e-3)
    gamma = (1.0 + 0.1 * rng.standard_normal(shape[-1])).astype(BF16)   # never uniform: hides index bugs
    return x, gamma


@pytest.mark.parametrize("shape", [(5, 128), (3, 20, 256), (33, 768), (100, 1024), (64, 2048), (17, 4096), (9, 8192)])
@pytest.mark.parametrize("pure", [False, True])
def test_forward_bit_exact_given_rnorm(shape, pure):
    from train_gpt_b200 import ops
    eps = 1e-6
    x, gamma = _inputs(shape, 11, eps)
    y, rn = ops.rmsnorm_fwd(to_torch_bf16(x), to_torch_bf16(gamma), eps, pure=pure, want_rnorm=True)
    rn = rn.cpu().numpy()[..., None]
    assert _ulp_diff_f32(rn, no.rnorm_of(x, eps)).max() <= 2
    ref = (no.rms_norm_pure if pure else no.rms_norm)(x, gamma, eps, rnorm=rn)
    assert np.array_equal(from_torch_bf16(y).view(np.uint16), ref.view(np.uint16))


def test_pure_norm_matches_reference_vectors(golden):
    from train_gpt_b200 import kernels
    x = np.asarray(golden["norm_x"]).view(BF16)
    gamma = np.asarray(golden["norm_gamma"]).view(BF16)
    y = kernels._rms_norm_pure(to_torch_bf16(x), to_torch_bf16(gamma), float(golden["norm_eps"]))
    got = from_torch_bf16(y).view(np.uint16)
    # the fixture's rnorm comes from a float64 variance; allow the rare last-bit rnorm flip
    assert (got != golden["norm_pure_y"]).mean() < 2e-3
    d = np.abs(got.view(BF16).astype(np.float32) - np.asarray(golden["norm_pure_y"]).view(BF16).astype(np.float32))
    assert (d <= 2.0 ** -7 * np.abs(got.view(BF16).astype(np.float32)) + 1e-30).all()


@pytest.mark.parametrize("shape", [(5, 128), (3, 20, 256), (100, 1024), (64, 2048), (9, 8192), (7, 384)])
@pytest.mark.parametrize("pure", [False, True])
def test_fused_norm_quant_bit_exact_given_rnorm(shape, pure):
    from train_gpt_b200 import ops
    eps = 1e-6
    x, gamma = _inputs(shape, 13, eps)
    q, s, y, rn = ops.rmsnorm_quant_fwd(to_torch_bf16(x), to_torch_bf16(gamma), eps, pure=pure, want_y=True, want_rnorm=True)
    rn = rn.cpu().numpy()[..., None]
    assert _ulp_diff_f32(rn, no.rnorm_of(x, eps)).max() <= 2
    q_ref, s_ref, y_ref = no.rmsnorm_quant(x, gamma, eps, rnorm=rn, pure=pure)
    assert np.array_equal(from_torch_bf16(y).view(np.uint16), y_ref.view(np.uint16))
    assert np.array_equal(f8_bytes(q), q_ref.view(np.uint8))
    assert np.array_equal(s.cpu().numpy().view(np.uint32), s_ref.view(np.uint32))
    # against the oracle's own rnorm: byte match rate (reported, loosely bounded)
    q_own, s_own, _ = no.rmsnorm_quant(x, gamma, eps, pure=pure)
    assert (f8_bytes(q) != q_own.view(np.uint8)).mean() < 5e-3
    # without the optional outputs the bytes are the same
    q2, s2, y2, rn2 = ops.rmsnorm_quant_fwd(to_torch_bf16(x), to_torch_bf16(gamma), eps, pure=pure)
    assert y2 is None and rn2 is None and torch.equal(q2.view(torch.uint8), q.view(torch.uint8)) and torch.equal(s2, s)


def test_fused_equals_norm_then_quantise_kernels():
    """The fused kernel against the two-kernel composition on a config-1-sized input."""
    from train_gpt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(32768, 2048, device="cuda", generator=g)
    x = torch.where(torch.rand(x.shape, device="cuda", generator=g) < 1e-3, x * 50, x).to(torch.bfloat16)
    gamma = (1 + 0.1 * torch.randn(2048, device="cuda", generator=g)).to(torch.bfloat16)
    q, s, _, _ = ops.rmsnorm_quant_fwd(x, gamma, 1e-6)
    y = ops.rmsnorm_fwd(x, gamma, 1e-6)
    q2, s2 = ops.quantize_rowwise(y)
    assert torch.equal(q.view(torch.uint8), q2.view(torch.uint8)) and torch.equal(s, s2)


@pytest.mark.parametrize("shape", [(5, 128), (3, 20, 256), (33, 768), (700, 1024), (40, 1280), (50, 1792), (3000, 2048),
                                   (17, 4096), (9, 8192)])
def test_backward(shape):
    from train_gpt_b200 import ops
    eps = 1e-5
    x, gamma = _inputs(shape, 17, eps)
    gy = normal_bf16(np.random.default_rng(3), shape)
    dx, dgamma = ops.rmsnorm_bwd(to_torch_bf16(x), to_torch_bf16(gamma), to_torch_bf16(gy), eps)
    dx_ref, dgamma_ref = no.rms_norm_bwd(x, gamma, gy, eps)
    a, b = from_torch_bf16(dx).astype(np.float32), dx_ref.astype(np.float32)
    # one bf16 ulp, plus the float32 cancellation error of gs - normed*dot on near-zero results
    tol = np.abs(b) * 2.0 ** -7 + np.sqrt(np.mean(b * b)) * 2.0 ** -14
    assert (np.abs(a - b) <= tol).all() and (a != b).mean() < 1e-2
    dg, dg_ref = from_torch_bf16(dgamma).astype(np.float32), dgamma_ref.astype(np.float32)
    assert np.abs(dg - dg_ref).max() <= 2.0 ** -7 * np.sqrt(np.mean(dg_ref ** 2)) + 2.0 ** -7 * np.abs(dg_ref).max()


@pytest.mark.parametrize("shape", [(5, 128), (3, 20, 256), (33, 768), (700, 1024), (40, 1280), (300, 2048)])
@pytest.mark.parametrize("pure", [False, True])
def test_residual_add_folded_into_the_norm(shape, pure):
    """tg_add_rmsnorm_quant_fwd: the sum equals the elementwise bf16 add bit for bit, and every other output
    equals tg_rmsnorm_quant_fwd of that sum bit for bit; without a quantised consumer only y is produced."""
    from train_gpt_b200 import ops
    eps = 1e-5
    x, gamma = _inputs(shape, 23, eps)
    res = normal_bf16(np.random.default_rng(5), shape, std=0.3)
    xt, rt, gt = to_torch_bf16(x), to_torch_bf16(res), to_torch_bf16(gamma)
    s, q, sc, y = ops.add_rmsnorm_quant_fwd(xt, rt, gt, eps, pure=pure)
    s_ref = xt + rt
    assert torch.equal(s.view(torch.int16), s_ref.view(torch.int16))
    q2, sc2, y2, _ = ops.rmsnorm_quant_fwd(s_ref, gt, eps, pure=pure, want_y=True)
    assert torch.equal(q.view(torch.uint8), q2.view(torch.uint8)) and torch.equal(sc, sc2)
    assert torch.equal(y.view(torch.int16), y2.view(torch.int16))
    s3, q3, sc3, y3 = ops.add_rmsnorm_quant_fwd(xt, rt, gt, eps, pure=pure, want_q=False)
    assert q3 is None and sc3 is None and torch.equal(y3.view(torch.int16), y2.view(torch.int16))
    assert torch.equal(s3.view(torch.int16), s_ref.view(torch.int16))
    with pytest.raises(ValueError):
        ops.add_rmsnorm_quant_fwd(xt, rt, gt, eps, want_q=False, want_y=False)


def test_residual_add_rejects_wide_rows():
    from train_gpt_b200 import ops
    x = torch.zeros((4, 4096), dtype=torch.bfloat16, device="cuda")
    g = torch.ones((4096,), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ValueError):
        ops.add_rmsnorm_quant_fwd(x, x, g, 1e-5)
    with pytest.raises(ValueError):
        ops.rmsnorm_bwd(x, g, x, 1e-5, addend=x)


@pytest.mark.parametrize("shape", [(5, 128), (3, 20, 256), (33, 768), (700, 1024), (40, 1280), (3000, 2048)])
def test_backward_with_the_skip_gradient_added(shape):
    """tg_rmsnorm_bwd_add: dgamma bit-equal to tg_rmsnorm_bwd; dx = bf16(addend + the unrounded input gradient),
    i.e. within half a bf16 ulp (of the sum) plus the plain kernel's own tolerance of addend + oracle dx."""
    from train_gpt_b200 import ops
    eps = 1e-5
    x, gamma = _inputs(shape, 17, eps)
    gy = normal_bf16(np.random.default_rng(3), shape)
    ad = normal_bf16(np.random.default_rng(4), shape, std=0.5)
    xt, gt, gyt, adt = to_torch_bf16(x), to_torch_bf16(gamma), to_torch_bf16(gy), to_torch_bf16(ad)
    dx_plain, dgamma_plain = ops.rmsnorm_bwd(xt, gt, gyt, eps)
    dx, dgamma = ops.rmsnorm_bwd(xt, gt, gyt, eps, addend=adt)
    assert torch.equal(dgamma.view(torch.int16), dgamma_plain.view(torch.int16))
    dx_ref, _ = no.rms_norm_bwd(x, gamma, gy, eps)
    want = ad.astype(np.float32) + dx_ref.astype(np.float32)
    got = from_torch_bf16(dx).astype(np.float32)
    b = dx_ref.astype(np.float32)
    tol = np.abs(want) * 2.0 ** -8 + np.abs(b) * 2.0 ** -7 + np.sqrt(np.mean(b * b)) * 2.0 ** -14
    assert (np.abs(got - want) <= tol).all()
    # and against the two-launch composition on the device: the same value up to the extra rounding of dx
    two = from_torch_bf16(adt + dx_plain).astype(np.float32)
    assert (np.abs(got - two) <= np.abs(two) * 2.0 ** -7 + np.abs(b) * 2.0 ** -8 + 1e-30).all()


@pytest.mark.parametrize("cols", [128, 384, 512, 1024, 2048])
def test_the_skip_gradient_is_added_to_the_rounded_product(cols):
    """dx = bf16(f32(f32(rnorm * (gs - normed * dot)) + addend)): two float32 roundings, not one.  Constant rows c with
    eps = 0 have rnorm = RN(1/c) and normed = 1 exactly, an upstream gradient of pairs (v, -v) has dot = 0 exactly, so dx is known to the
    bit whatever the order of the sums; where the addend cancels the product's leading bits, the two forms differ."""
    from train_gpt_b200 import ops
    c = np.arange(128, 256, dtype=np.float32) / 64.0
    rn = (1.0 / c.astype(np.float64)).astype(np.float32)
    ok = c * rn == 1.0
    c, rn = c[ok], rn[ok]
    rows = len(c)
    rng = np.random.default_rng(cols)
    v = rng.integers(1, 256, (rows, cols // 2)).astype(np.float32) / 128.0
    g = np.stack((v, -v), axis=2).reshape(rows, cols)
    exact = rn[:, None].astype(np.float64) * g                       # 32 bits: exact in float64
    a = (-exact).astype(np.float32).astype(BF16)
    want = (exact.astype(np.float32) + a.astype(np.float32)).astype(BF16)
    fused = (exact + a.astype(np.float64)).astype(np.float32).astype(BF16)
    assert (want != fused).sum() >= 8
    dx, _ = ops.rmsnorm_bwd(to_torch_bf16(np.broadcast_to(c[:, None], g.shape)), to_torch_bf16(np.ones(cols)), to_torch_bf16(g), 0.0,
                            addend=to_torch_bf16(a))
    assert np.array_equal(from_torch_bf16(dx).astype(np.float32), want.astype(np.float32))


def _weight_gradient(partial):
    """The norm-weight gradient of (blocks, cols) float32 partial sums, added in the order that the kernel states."""
    n = len(partial)
    total = None
    for w in range(8):
        s = np.zeros((4, partial.shape[1]), np.float32)
        b = w
        while b + 24 < n:
            for i in range(4):
                s[i] += partial[b + 8 * i]
            b += 32
        for b in range(b, n, 8):
            s[0] += partial[b]
        u = (s[0] + s[1]) + (s[2] + s[3])
        total = u if total is None else total + u
    return total.astype(BF16)


@pytest.mark.parametrize("blocks", [1, 7, 8, 24, 25, 31, 33, 57, 96, 121, 147, 148])
@pytest.mark.parametrize("cols", [128, 1000])
def test_order_of_the_weight_gradients_sums(blocks, cols):
    """dgamma is the sum of the thread blocks' partial sums in an order that depends on their number alone, to the bit: another
    order is another last bit, which a training run amplifies."""
    from train_gpt_b200 import _lib
    lib = _lib.load()
    per_block = 16 if cols <= 512 else 12
    rows = per_block * (blocks - 1) + 3
    x, gamma = _inputs((rows, cols), blocks, 1e-6)
    gy = normal_bf16(np.random.default_rng(blocks), (rows, cols), std=30.0)
    x[-1] = 1.0                              # the last row takes the columns' sums back, so that their last bits show in bf16
    wide = x.astype(np.float64)
    normed = wide / np.sqrt((wide * wide).mean(1, keepdims=True) + 1e-6)
    gy[-1] = -(gy[:-1].astype(np.float64) * normed[:-1]).sum(0)
    t = [to_torch_bf16(v) for v in (x, gamma, gy)]
    need = lib.tg_rmsnorm_bwd_scratch_bytes(rows, cols)
    assert need == blocks * cols * 4
    partial = torch.zeros((blocks, cols), device="cuda")
    dx, dgamma = torch.empty_like(t[0]), torch.empty_like(t[1])
    _lib.check(lib.tg_rmsnorm_bwd(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), 1e-6, dx.data_ptr(), dgamma.data_ptr(),
                                  partial.data_ptr(), rows, cols, torch.cuda.current_stream().cuda_stream), "tg_rmsnorm_bwd")
    assert np.array_equal(from_torch_bf16(dgamma).view(np.uint16), _weight_gradient(partial.cpu().numpy()).view(np.uint16))


def test_backward_matches_reference_vectors_and_autograd(golden):
    from train_gpt_b200 import kernels
    x = to_torch_bf16(np.asarray(golden["norm_x"]).view(BF16)).requires_grad_(True)
    gamma = to_torch_bf16(np.asarray(golden["norm_gamma"]).view(BF16)).requires_grad_(True)
    gy = to_torch_bf16(np.asarray(golden["norm_gy"]).view(BF16))
    y = kernels.rms_norm(x, gamma, float(golden["norm_eps"]))
    y.backward(gy)
    dx = from_torch_bf16(x.grad).astype(np.float32)
    ref = np.asarray(golden["norm_dx"]).view(BF16).astype(np.float32)
    assert (np.abs(dx - ref) <= np.abs(ref) * 2.0 ** -7 + 1e-30).all() and (dx != ref).mean() < 1e-2
    dg = from_torch_bf16(gamma.grad).astype(np.float32)
    dg_ref = np.asarray(golden["norm_dgamma"]).view(BF16).astype(np.float32)
    assert np.abs(dg - dg_ref).max() <= 2.0 ** -6 * np.abs(dg_ref).max()
    assert x.grad.dtype == torch.bfloat16 and gamma.grad.shape == (256,)


@pytest.mark.parametrize("rows,cols", [(8200, 128), (4100, 384), (1030, 1024), (700, 2048), (500, 2176), (460, 2560), (401, 3000), (371, 4096),
                                       (301, 4352), (150, 5640), (180, 6144), (160, 6656), (155, 7040), (140, 8192)])
@pytest.mark.parametrize("pure", [False, True])
def test_every_split_of_a_row_over_warps(rows, cols, pure):
    """Enough rows for the kernels that give one to eight warps to a row (fewer take a block per row): every number of chunks per
    warp, whole and ragged, forward, quantised and backward, against the oracle."""
    from train_gpt_b200 import ops
    eps = 1e-6
    x, gamma = _inputs((rows, cols), rows, eps)
    xt, gt = to_torch_bf16(x), to_torch_bf16(gamma)
    y, rn = ops.rmsnorm_fwd(xt, gt, eps, pure=pure, want_rnorm=True)
    rn = rn.cpu().numpy()[..., None]
    assert _ulp_diff_f32(rn, no.rnorm_of(x, eps)).max() <= 2
    ref = (no.rms_norm_pure if pure else no.rms_norm)(x, gamma, eps, rnorm=rn)
    assert np.array_equal(from_torch_bf16(y).view(np.uint16), ref.view(np.uint16))
    if cols % 128 == 0:
        q, s, y2, _ = ops.rmsnorm_quant_fwd(xt, gt, eps, pure=pure, want_y=True)
        q_ref, s_ref = ops.quantize_rowwise(y)
        assert torch.equal(y2, y) and torch.equal(q.view(torch.uint8), q_ref.view(torch.uint8)) and torch.equal(s, s_ref)
    if not pure:
        test_backward((rows, cols))


# the largest tensors that take a block per row, and one row more, which takes warps: rows of one, two and four groups of pieces, a group
# that is not full, the widest
@pytest.mark.parametrize("rows,cols", [(1024, 1024), (2048, 1536), (1536, 2048), (910, 2304), (682, 3072), (444, 4608), (409, 5120), (256, 8192), (291, 7168), (296, 6144)])
def test_block_per_row_has_the_bits_of_warps_per_row(rows, cols):
    from train_gpt_b200 import ops
    gen = torch.Generator("cuda").manual_seed(cols)
    x = torch.randn(rows + 400, cols, device="cuda", generator=gen).to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(cols, device="cuda", generator=gen)).to(torch.bfloat16)
    for pure in (False, True):
        few = ops.rmsnorm_quant_fwd(x[:rows], w, 1e-6, pure, want_y=True, want_rnorm=True)
        many = ops.rmsnorm_quant_fwd(x, w, 1e-6, pure, want_y=True, want_rnorm=True)
        for a, b in zip(few, many):
            assert torch.equal(a.view(torch.uint8), b[:rows].view(torch.uint8))
        assert torch.equal(ops.rmsnorm_fwd(x[:rows], w, 1e-6, pure), many[2][:rows])
