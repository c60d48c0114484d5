"""The kernel with the scale ring.  On pairs of SMs it is compared with the other tiled kernel: a row (or column) of the result depends on
its own operands only and is summed in the same order by either, so a problem computed in slices too small for pairs has the same
bits.  On single SMs it is compared with the product in float64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
SINGLE, PAIRS = 1, 2


def _plan(M, N, K, major, gran):
    from train_gpt_b200 import _lib
    mn = _lib.TG_MAJOR_MN
    args = _lib.GemmArgs(M=M, N=N, K=K, lda=(M if major == mn else K) + 15 & ~15, ldb=N + 15 & ~15, a_major=major, b_major=mn, sb_gran_n=gran, sb_stride_n=1, ldd=N)
    kernel = ctypes.c_int(-1)
    rc = _lib.load().tgh_gemm_kernel(ctypes.byref(args), ctypes.byref(kernel))
    return kernel.value if rc == _lib.TG_OK else -1            # (-1: the few-token kernel's)


def _f8(gen, *shape):
    return (torch.randn(*shape, device="cuda", generator=gen) * 60).to(torch.float8_e4m3fn)


def _scales(gen, *shape):
    return torch.rand(*shape, device="cuda", generator=gen) * 3 - 1


# rows: whole tiles, one row in the last pair, none or a few in its second CTA, a second CTA one row short; columns: whole tiles, a
# ragged last one, one that ends in the first half; contraction: one block more than the stages, odd, many
@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,K,N,tile", [(4096, 1024, 4096, (128, 128)), (6145, 640, 2048, (128, 128)), (6145 + 128, 1152, 2048, (128, 1)),
                                         (5000, 1024, 4104, (128, 1)), (8191, 128, 2688, (128, 128)), (8191, 384, 2304 + 136, (128, 1)),
                                         (3000, 2048, 4096, (128, 128))])
def test_forward_has_the_bits_of_its_slices(M, K, N, tile, out):
    from train_gpt_b200 import _lib, ops
    gen = torch.Generator("cuda").manual_seed(M + N)
    a, sa = _f8(gen, M, K), _scales(gen, M, K // 128)
    w = _f8(gen, K, N + 15 & ~15)[:, :N]
    sw = _scales(gen, K // 128, N if tile == (128, 1) else N // 128)
    gran = 1 if tile == (128, 1) else 128
    kw = dict(N=N, K=K, a_major=_lib.TG_MAJOR_K, b_major=_lib.TG_MAJOR_MN, sa_strides=(sa.stride(0), 1), sb_strides=(1, sw.stride(0)), sb_gran_n=gran, out_dtype=out, split=False)
    assert _plan(M, N, K, _lib.TG_MAJOR_K, gran) == PAIRS
    status = ops.new_status("cuda")
    y = ops.gemm_blockscaled(a, w, sa, sw, M=M, status=status, **kw)
    for r in range(0, M, 512):
        m = min(512, M - r)
        assert _plan(m, N, K, _lib.TG_MAJOR_K, gran) != PAIRS
        if m <= 128:
            continue               # (the few-token kernel adds in another order)
        assert torch.equal(y[r:r + m], ops.gemm_blockscaled(a[r:r + m], w, sa[r:r + m], sw, M=m, status=status, **kw)), r
    if M % 512 and M % 512 <= 128:
        ref = (a[M - 1:].float().view(-1, 128) * sa[M - 1:].view(-1, 1)).view(1, K).double() @ (
            w.double() * (sw if gran == 1 else sw.repeat_interleave(128, 1)).double().repeat_interleave(128, 0))
        assert (y[M - 1:].double() - ref).norm() < 4e-3 * ref.norm()
    assert int(status.item()) == 0


# tokens: ragged blocks (zeros past the end), fewer blocks than stages; outputs: a ragged last tile each way
@pytest.mark.parametrize("T,K,N", [(600, 8192, 2048), (1000, 4096, 4096), (300, 2176, 8192 + 136), (1030, 8192, 2048)])
def test_weight_gradient_has_the_bits_of_its_slices(T, K, N):
    from train_gpt_b200 import _lib, ops
    gen = torch.Generator("cuda").manual_seed(T)
    x, g = _f8(gen, T, K), _f8(gen, T, N + 15 & ~15)[:, :N]
    tb = (T + 127) // 128
    sx, sg = _scales(gen, tb, K), _scales(gen, tb, N)
    kw = dict(N=N, K=T, a_major=_lib.TG_MAJOR_MN, b_major=_lib.TG_MAJOR_MN, sa_strides=(1, sx.stride(0)), sb_strides=(1, N), sb_gran_n=1, split=False)
    assert _plan(K, N, T, _lib.TG_MAJOR_MN, 1) == PAIRS
    status = ops.new_status("cuda")
    dw = ops.gemm_blockscaled(x, g, sx, sg, M=K, status=status, **kw)
    for r in range(0, K, 384):
        m = min(384, K - r)
        assert _plan(m, N, T, _lib.TG_MAJOR_MN, 1) != PAIRS
        xs = x[:, r:r + m].contiguous()
        part = ops.gemm_blockscaled(xs, g, sx[:, r:r + m].contiguous(), sg, M=m, status=status, **dict(kw, sa_strides=(1, m)))
        assert torch.equal(dw[r:r + m], part), r
    assert int(status.item()) == 0


def _close(y, ref):
    """One rounding to the output type, and float32 sums of at most 128 blocks of 128 products."""
    ulp = 2.0 ** -8 if y.dtype == torch.bfloat16 else 0.0
    assert bool(((y.double() - ref).abs() <= ulp * ref.abs() + 1e-5 * ref.square().mean().sqrt()).all())


# 128-column tiles (two of them wider than N), 192-column tiles (a ragged last one); twelve blocks, more than the ring, one past it
@pytest.mark.parametrize("M,K,N,out", [(200, 1536, 1000, torch.bfloat16), (129, 1664, 8192, torch.float32), (1000, 2048, 136, torch.bfloat16),
                                        (1100, 1792, 2952, torch.bfloat16), (640, 4096, 4096, torch.bfloat16)])
def test_column_scales_on_single_sms_forward(M, K, N, out):
    from train_gpt_b200 import _lib, ops
    gen = torch.Generator("cuda").manual_seed(K)
    a, sa = _f8(gen, M, K), _scales(gen, M, K // 128)
    w, sw = _f8(gen, K, N + 15 & ~15)[:, :N], _scales(gen, K // 128, N)
    if M % 128:
        assert _plan(M, N, K, _lib.TG_MAJOR_K, 1) == SINGLE
    status = ops.new_status("cuda")
    y = ops.gemm_blockscaled(a, w, sa, sw, M=M, N=N, K=K, a_major=_lib.TG_MAJOR_K, b_major=_lib.TG_MAJOR_MN, sa_strides=(K // 128, 1),
                             sb_strides=(1, N), sb_gran_n=1, out_dtype=out, status=status)
    _close(y, (a.double() * sa.double().repeat_interleave(128, 1)) @ (w.double() * sw.double().repeat_interleave(128, 0)))
    assert int(status.item()) == 0


@pytest.mark.parametrize("T,K,N", [(1537, 256, 384), (4096, 768, 3072), (2000, 1024, 1160), (1700, 128, 200)])
def test_column_scales_on_single_sms_weight_gradient(T, K, N):
    from train_gpt_b200 import _lib, ops
    gen = torch.Generator("cuda").manual_seed(T)
    x, g = _f8(gen, T, K), _f8(gen, T, N + 15 & ~15)[:, :N]
    tb = (T + 127) // 128
    sx, sg = _scales(gen, tb, K), _scales(gen, tb, N)
    assert _plan(K, N, T, _lib.TG_MAJOR_MN, 1) == SINGLE
    status = ops.new_status("cuda")
    dw = ops.gemm_blockscaled(x, g, sx, sg, M=K, N=N, K=T, a_major=_lib.TG_MAJOR_MN, b_major=_lib.TG_MAJOR_MN, sa_strides=(1, K), sb_strides=(1, N),
                              sb_gran_n=1, status=status)
    _close(dw, (x.double() * sx.double().repeat_interleave(128, 0)[:T]).t() @ (g.double() * sg.double().repeat_interleave(128, 0)[:T]))
    assert int(status.item()) == 0


def test_two_streams_and_a_graph():
    """Launches on two streams at once, and replayed: no state is shared between them."""
    from train_gpt_b200 import ops
    gen = torch.Generator("cuda").manual_seed(1)
    ops_ = []
    for _ in range(2):
        a, w = _f8(gen, 8192, 1024), _f8(gen, 1024, 4096)
        ops_.append((a, _scales(gen, 8192, 8), w, _scales(gen, 8, 32)))
    want = [ops.gemm_fwd(*o, (128, 128)) for o in ops_]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
    got = [None, None]
    for _ in range(5):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i] = ops.gemm_fwd(*ops_[i], (128, 128))
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = [ops.gemm_fwd(*o, (128, 128)) for o in ops_]
    for o in out:
        o.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(out, want))
    ops.check_status()
