"""A linear's data and weight gradient in one launch: the bits of the two launches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one tile each; ragged tokens; sizes that fit one wave together and, at the end, sizes that do not (two launches); the modes' three kinds of scales
ONE_WAVE = [(130, 128, 128), (1000, 384, 256), (1024, 512, 128), (700, 640, 768), (1024, 1152, 640), (1025, 1280, 640)]
APART = [(1024, 128, 17920), (300, 128, 4096)]
MODES = [((128, 128), "fp8"), ((128, 1), "fp8"), ((128, 128), "fp8_blockgrad")]


@pytest.mark.parametrize("tokens,k,n", ONE_WAVE + APART)
@pytest.mark.parametrize("tile,mode", MODES)
def test_backward_has_the_bits_of_two_launches(tokens, k, n, tile, mode):
    _compare(tokens, k, n, tile, mode)


# Both on pairs of SMs: a weight gradient cut in two, in three, uncut; several rounds of it, one, less than one; idle pairs that take all of
# the data gradient's tiles, a round of them, or none; ragged tokens and columns (an odd number of 128-column blocks).  With the rounds
# of data-gradient tiles that idle pairs take first.  The others stay apart.
ON_PAIRS = [(8192, 2048, 2048, 1), (5000, 2048, 4224, 0), (24576, 1024, 1024, 6), (5000, 1024, 4096, 0), (24576, 1024, 3072, 9), (2048, 2048, 2048, 0),
            (700, 4096, 4096, 0), (12000, 768, 3072, 3), (4100, 640, 3200, 1)]
PAIRS_APART = [(6145, 2048, 2176), (32768, 2048, 6144), (8466, 384, 256), (512, 1024, 1920)]


@pytest.mark.parametrize("tokens,k,n", [s[:3] for s in ON_PAIRS] + PAIRS_APART[:1])
def test_backward_on_pairs_has_the_bits_of_two_launches(tokens, k, n):
    _compare(tokens, k, n, (128, 128), "fp8")


def _compare(tokens, k, n, tile, mode):
    from train_gpt_b200 import fp8, ops
    gen = torch.Generator("cuda").manual_seed(tokens + k + n)
    x = torch.randn(tokens, k, device="cuda", generator=gen).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(k, n, device="cuda", generator=gen) * 0.05).to(torch.bfloat16).requires_grad_()
    g = torch.randn(tokens, n, device="cuda", generator=gen).to(torch.bfloat16)
    fp8.block_scaled_matmul(x, w, weight_tile=tile, backward=mode).backward(g)
    status = ops.new_status("cuda")
    x_q, x_s = ops.quantize_colwise(x.detach())
    g_q, g_s = ops.quantize_rowwise(g)
    w_q, w_s = ops.quantize_block128(w.detach()) if tile == (128, 128) else ops.quantize_rowwise(w.detach())
    grad_tile = (128, 128) if mode == "fp8_blockgrad" else (128, 1)
    c_q, c_s = ops.quantize_block128(g) if mode == "fp8_blockgrad" else ops.quantize_colwise(g)
    assert torch.equal(x.grad, ops.gemm_dgrad(g_q, g_s, w_q, w_s, tile, status=status))
    assert torch.equal(w.grad, ops.gemm_wgrad(x_q, x_s, c_q, c_s, grad_tile=grad_tile, status=status))
    assert int(status.item()) == 0
    ops.check_status()
