"""The rule that picks the GEMM's kernel, tile width and contraction ranges, on the CPU, against times measured on a B200 with each choice
forced (microseconds of single launches in a graph): what is taken is at most 4 % slower than the fastest."""
import ctypes

import pytest

# (what, tokens, K, N, scale per column, us with wide tiles, us with 128-column tiles, us on pairs of SMs)
MEASURED = [
    ("wgrad", 16, 8192, 8192, 1, 28.8, 31.7, 30.4),
    ("wgrad", 64, 8192, 8192, 1, 29.0, 31.9, 30.7),
    ("wgrad", 256, 8192, 8192, 1, 37.4, 42.0, 32.8),
    ("wgrad", 512, 8192, 8192, 1, 57.8, 62.9, 47.7),
    ("wgrad", 16, 2048, 8192, 1, 10.9, 12.3, 11.1),
    ("wgrad", 128, 4096, 4096, 1, 10.7, 10.8, 11.1),
    ("wgrad", 64, 1024, 4096, 1, 5.8, 4.8, 6.0),
    ("wgrad", 256, 2048, 2048, 1, 6.4, 5.3, 6.6),
    ("wgrad", 384, 3072, 3072, 1, 10.5, 9.5, 10.0),
    ("fwd", 8192, 256, 8192, 0, 31.8, 38.5, 33.9),
    ("fwd", 32768, 256, 1024, 0, 18.2, 21.4, 20.0),
    ("fwd", 4096, 256, 4096, 0, 11.5, 12.5, 11.9),
    ("fwd", 32768, 128, 8192, 0, 107.1, 112.9, 115.3),
    ("fwd", 32768, 512, 4096, 0, 84.9, 106.4, 73.6),
    ("fwd", 4096, 128, 1024, 0, 4.9, 4.5, 5.6),
    ("fwd", 4096, 512, 1024, 0, 6.3, 6.2, 7.2),
    ("fwd", 200, 1024, 8192, 0, 7.5, 5.9, 8.4),
    ("fwd", 4096, 2048, 4096, 0, 33.4, 41.2, 33.1),
    ("fwd", 32768, 128, 8192, 1, 103.7, 116.9, 107.6),
    ("fwd", 8192, 256, 8192, 1, 37.6, 42.3, 32.9),
    ("fwd", 8192, 512, 8192, 1, 57.9, 62.9, 47.3),
    ("fwd", 4096, 512, 1024, 1, 8.7, 6.9, 7.9),
    ("fwd", 200, 2048, 8192, 1, 11.9, 9.8, 14.0),
    ("dgrad", 8192, 8192, 256, 0, 31.8, 38.6, 34.0),
    ("dgrad", 32768, 8192, 128, 1, 103.0, 117.0, 107.5),
    ("dgrad", 4096, 1024, 512, 1, 8.7, 6.9, 8.0),
]


# Single SMs or pairs, with either forced: (what, tokens, K, N, scale per column, us on single SMs, us on pairs).  The data gradients with a scale
# per column have those apart in memory.  Contractions of one to 58 blocks, cut in up to eight ranges or not, half a wave of pairs and more.
PAIRS_MEASURED = [
    ("dgrad", 445, 4736, 3456, 1, 13.0, 21.0), ("dgrad", 269, 6144, 5888, 1, 23.1, 35.3), ("dgrad", 512, 2560, 2560, 1, 12.8, 16.1),
    ("dgrad", 7567, 384, 5760, 1, 28.4, 34.5), ("dgrad", 4992, 1024, 3584, 1, 31.0, 38.4), ("dgrad", 12753, 512, 5888, 1, 63.1, 69.4),
    ("dgrad", 738, 7680, 3712, 1, 32.9, 40.9), ("dgrad", 8035, 1280, 256, 1, 8.5, 10.2), ("dgrad", 21632, 384, 1664, 1, 22.6, 27.6),
    ("dgrad", 14464, 640, 2048, 1, 27.2, 33.0), ("dgrad", 29316, 384, 5376, 1, 100.5, 117.0), ("dgrad", 12416, 1664, 128, 1, 12.3, 14.5),
    ("dgrad", 310, 2688, 3200, 1, 13.2, 15.2), ("dgrad", 3328, 384, 3456, 1, 17.3, 18.8), ("dgrad", 1536, 3328, 1152, 1, 13.1, 15.3),
    ("dgrad", 1920, 1920, 5248, 1, 66.9, 42.4), ("dgrad", 5760, 640, 6656, 1, 89.2, 49.8), ("dgrad", 2176, 3328, 7168, 1, 160.9, 100.2),
    ("dgrad", 7168, 2560, 3712, 1, 97.4, 81.8), ("dgrad", 11779, 1536, 7424, 1, 195.1, 170.2), ("dgrad", 22016, 1280, 1280, 1, 53.9, 44.2),
    ("dgrad", 169, 4224, 6272, 1, 23.6, 20.8), ("dgrad", 1922, 768, 5248, 1, 28.1, 23.9), ("dgrad", 738, 5248, 4992, 1, 34.7, 31.7),
    ("dgrad", 24320, 5888, 256, 1, 78.4, 66.7), ("dgrad", 10439, 7552, 384, 1, 57.4, 48.0),
    ("fwd", 26276, 128, 4608, 0, 51.6, 55.0), ("fwd", 8589, 256, 4992, 0, 23.6, 25.0), ("fwd", 7674, 768, 7936, 0, 57.3, 51.0),
    ("fwd", 26775, 128, 768, 1, 12.3, 14.6), ("fwd", 9930, 128, 6144, 1, 27.4, 29.7), ("fwd", 20225, 768, 384, 1, 14.7, 16.5),
    ("fwd", 11541, 768, 3328, 1, 48.2, 41.0), ("fwd", 15295, 896, 1408, 1, 33.4, 28.6), ("fwd", 3897, 896, 3456, 1, 19.9, 21.0),
    ("dgrad", 20960, 896, 128, 0, 11.6, 14.1), ("dgrad", 5007, 7936, 256, 0, 22.3, 23.6), ("dgrad", 6193, 5248, 256, 0, 18.9, 20.3),
    ("dgrad", 27860, 4096, 512, 0, 74.8, 67.2), ("dgrad", 10615, 896, 768, 0, 12.2, 13.1),
    ("wgrad", 30720, 1408, 1664, 0, 95.2, 85.5), ("wgrad", 17716, 2688, 2944, 1, 200.2, 179.6), ("wgrad", 23680, 1920, 2304, 1, 150.9, 132.6),
    ("wgrad", 6016, 2176, 2048, 1, 48.5, 42.0), ("wgrad", 24190, 384, 1152, 1, 21.7, 37.9), ("wgrad", 19455, 640, 1792, 1, 33.1, 48.4),
    ("fwd", 8192, 128, 3072, 1, 13.6, 16.5), ("fwd", 8192, 256, 3072, 1, 16.4, 17.7), ("fwd", 8192, 256, 4096, 1, 21.8, 19.7), ("wgrad", 256, 4096, 4096, 1, 12.8, 12.1), ("wgrad", 256, 3584, 5632, 1, 14.6, 15.8), ("wgrad", 384, 5120, 5120, 1, 23.3, 20.2),
    ("fwd", 303, 6016, 1408, 1, 12.6, 15.3), ("fwd", 2304, 7680, 896, 1, 29.6, 35.7), ("dgrad", 515, 2176, 8064, 0, 19.3, 29.7),
    ("fwd", 1152, 5248, 1920, 0, 19.8, 29.8),
]

# The few-token kernel or the tiled ones: (tokens, K, N, scale per column, us of the few-token kernel, us of the tiled ones)
FEW_MEASURED = [
    (1, 2048, 256, 1, 5.0, 7.4), (16, 2560, 512, 0, 7.1, 8.1), (16, 3072, 512, 0, 7.3, 6.7), (16, 8192, 256, 0, 12.5, 7.5), (16, 16384, 512, 0, 9.0, 10.0),
    (16, 32768, 256, 0, 12.2, 14.3), (32, 3584, 512, 0, 6.2, 7.4), (32, 512, 512, 0, 4.0, 3.8), (48, 1024, 4096, 0, 6.3, 5.7), (64, 2048, 512, 0, 5.8, 7.1),
    (65, 2048, 2176, 0, 7.0, 7.8), (100, 1024, 4096, 0, 7.5, 5.8), (100, 1024, 4096, 1, 7.5, 6.2), (100, 4096, 4096, 0, 10.8, 10.1),
    (100, 8192, 4096, 0, 14.4, 14.9), (100, 5504, 5120, 0, 13.2, 13.7), (128, 8192, 3072, 0, 13.1, 14.4), (128, 5504, 4096, 0, 12.6, 14.3),
    (128, 4096, 6144, 0, 13.9, 13.5),
]


@pytest.fixture(scope="module")
def lib():
    from train_gpt_b200 import build, _lib
    build.build()
    return _lib.load()


def _args(what, tokens, k, n, columns):
    """A linear's product as the library's callers lay it out."""
    from train_gpt_b200 import _lib
    major, mn = _lib.TG_MAJOR_K, _lib.TG_MAJOR_MN
    if what == "wgrad":
        return _lib.GemmArgs(M=k, N=n, K=tokens, lda=(k + 15) // 16 * 16, ldb=n, a_major=mn, b_major=mn, sb_gran_n=1 if columns else 128,
                             sb_stride_n=1, ldd=n)
    if what == "fwd":
        return _lib.GemmArgs(M=tokens, N=n, K=k, lda=k, ldb=n, a_major=major, b_major=mn, sb_gran_n=1 if columns else 128, sb_stride_n=1, ldd=n)
    return _lib.GemmArgs(M=tokens, N=k, K=n, lda=n, ldb=n, a_major=major, b_major=major, sb_gran_n=1 if columns else 128, sb_stride_n=n // 128, ldd=k)


def _plan(lib, what, tokens, k, n, columns):
    from train_gpt_b200 import _lib
    args = _args(what, tokens, k, n, columns)
    width, ranges = ctypes.c_int(), ctypes.c_int()
    assert lib.tgh_gemm_plan(ctypes.byref(args), ctypes.byref(width), ctypes.byref(ranges)) == _lib.TG_OK
    return width.value, ranges.value


def _kernel(lib, what, tokens, k, n, columns):
    kernel = ctypes.c_int()
    assert lib.tgh_gemm_kernel(ctypes.byref(_args(what, tokens, k, n, columns)), ctypes.byref(kernel)) == 0
    return kernel.value


@pytest.mark.parametrize("what,tokens,k,n,columns,wide_us,narrow_us,pair_us", MEASURED)
def test_takes_the_faster_width(lib, what, tokens, k, n, columns, wide_us, narrow_us, pair_us):
    width, ranges = _plan(lib, what, tokens, k, n, columns)
    assert width in (128, 192, 256) and ranges == 1
    on_pairs = _kernel(lib, what, tokens, k, n, columns) == 2
    assert (pair_us if on_pairs else narrow_us if width == 128 else wide_us) <= 1.04 * min(wide_us, narrow_us, pair_us), (width, on_pairs)


@pytest.mark.parametrize("tokens,k,n,columns,few_us,tiled_us", FEW_MEASURED)
def test_takes_the_few_token_kernel_where_it_is_faster(lib, tokens, k, n, columns, few_us, tiled_us):
    from train_gpt_b200 import _lib
    width, ranges = ctypes.c_int(), ctypes.c_int()
    rc = lib.tgh_gemm_plan(ctypes.byref(_args("fwd", tokens, k, n, columns)), ctypes.byref(width), ctypes.byref(ranges))
    assert rc in (_lib.TG_OK, _lib.TG_ERR_TOO_LARGE)
    assert (tiled_us if rc == _lib.TG_OK else few_us) <= 1.03 * min(few_us, tiled_us)


@pytest.mark.parametrize("what,tokens,k,n,columns,single_us,pair_us", PAIRS_MEASURED)
def test_takes_the_faster_of_single_sms_and_pairs(lib, what, tokens, k, n, columns, single_us, pair_us):
    assert (pair_us if _kernel(lib, what, tokens, k, n, columns) == 2 else single_us) <= 1.04 * min(single_us, pair_us)


# The scale ring on single SMs: (what, tokens, K, N, us without, us with)
@pytest.mark.parametrize("what,tokens,k,n,plain_us,ring_us", [("wgrad", 12026, 384, 256, 10.36, 10.65), ("wgrad", 2944, 640, 384, 9.39, 9.64),
                                                              ("wgrad", 12928, 256, 768, 11.8, 12.1), ("wgrad", 15047, 2176, 256, 20.0, 18.2),
                                                              ("wgrad", 16896, 1792, 128, 15.2, 14.6), ("dgrad", 19200, 128, 6656, 65.5, 53.4),
                                                              ("wgrad", 1920, 768, 384, 8.35, 7.92), ("dgrad", 244, 1152, 1792, 9.7, 7.7)])
def test_takes_the_scale_ring_where_it_is_faster(lib, what, tokens, k, n, plain_us, ring_us):
    kernel = _kernel(lib, what, tokens, k, n, 1)
    assert kernel in (0, 1) and (ring_us if kernel == 1 else plain_us) <= 1.02 * min(plain_us, ring_us)


@pytest.mark.parametrize("what,tokens,k,n,ranges", [("wgrad", 8192, 1024, 1024, 3), ("wgrad", 8192, 1024, 4096, 2), ("wgrad", 8192, 4096, 1024, 2),
                                                    ("wgrad", 8192, 1024, 3072, 1), ("wgrad", 32768, 1024, 1024, 3),
                                                    ("fwd", 8192, 1024, 4096, 1), ("dgrad", 1024, 128, 512, 1)])
def test_a_training_steps_contraction_ranges(lib, what, tokens, k, n, ranges):
    """The number of ranges shows in the last bit of a weight gradient, so it does not change for whole blocks of tokens."""
    assert _plan(lib, what, tokens, k, n, what == "wgrad")[1] == ranges


def test_pairs_leave_reserved_sms_room_wherever_their_blocks_lie(lib):
    """A block of another kernel on one SM of a pair keeps the pair waiting until that kernel ends: with n SMs reserved a launch takes n pairs
    fewer, and a problem that this leaves too few goes to single SMs."""
    from train_gpt_b200 import _lib
    args = _lib.GemmArgs(M=32768, N=6144, K=2048, lda=2048, ldb=6144, a_major=_lib.TG_MAJOR_K, b_major=_lib.TG_MAJOR_MN, sb_gran_n=128, ldd=6144)
    kernel = ctypes.c_int()
    before = lib.tg_set_gemm_reserved_sms(0)
    try:
        for reserved, on_pairs in ((0, True), (8, True), (64, False)):
            lib.tg_set_gemm_reserved_sms(reserved)
            assert lib.tgh_gemm_kernel(ctypes.byref(args), ctypes.byref(kernel)) == _lib.TG_OK
            assert (kernel.value == 2) == on_pairs, reserved
        lib.tg_set_gemm_reserved_sms(0)
        all_pairs = lib.tgh_gemm_pairs()
        lib.tg_set_gemm_reserved_sms(8)
        assert lib.tgh_gemm_pairs() == all_pairs - 8
    finally:
        lib.tg_set_gemm_reserved_sms(before)


def _joint(lib, tokens, k, n, tile, mode):
    """How a linear's backward pass runs its two products: tgh_gemm_two_plan's answer and rounds."""
    from train_gpt_b200 import _lib
    major, mn, columns, g_columns = _lib.TG_MAJOR_K, _lib.TG_MAJOR_MN, tile == (128, 1), mode == "fp8"
    dgrad = _lib.GemmArgs(M=tokens, N=k, K=n, lda=n, ldb=n, a_major=major, b_major=major, sa_stride_m=n // 128, sa_stride_kb=1,
                          sb_stride_n=n // 128, sb_stride_kb=1, sb_gran_n=1 if columns else 128, ldd=k)
    wgrad = _lib.GemmArgs(M=k, N=n, K=tokens, lda=k, ldb=n, a_major=mn, b_major=mn, sa_stride_m=1, sa_stride_kb=k, sb_stride_n=1,
                          sb_stride_kb=n if g_columns else n // 128, sb_gran_n=1 if g_columns else 128, ldd=n)
    for args in (dgrad, wgrad):
        args.workspace_bytes = lib.tg_gemm_workspace_bytes(ctypes.byref(args))
        args.workspace = 4096 if args.workspace_bytes else None            # (never read here)
    rounds = ctypes.c_int()
    return lib.tgh_gemm_two_plan(ctypes.byref(dgrad), ctypes.byref(wgrad), ctypes.byref(rounds)), rounds.value


def test_two_products_run_as_their_gpu_tests_say(lib):
    """The sizes that test_gpu_gemm_two compares with two launches do take one, and the launch that they stand for."""
    from test_gpu_gemm_two import APART, MODES, ON_PAIRS, ONE_WAVE, PAIRS_APART
    for tile, mode in MODES:
        assert {_joint(lib, *s, tile, mode) for s in ONE_WAVE} == {(1, 0)}
        assert {_joint(lib, *s, tile, mode) for s in APART} == {(0, 0)}
    assert [_joint(lib, *s[:3], (128, 128), "fp8") for s in ON_PAIRS] == [(2, s[3]) for s in ON_PAIRS]
    assert {_joint(lib, *s, (128, 128), "fp8") for s in PAIRS_APART} == {(0, 0)}
