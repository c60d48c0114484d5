"""The rule that picks the loss's kernel for ragged rows, on the CPU, against times measured on a B200 with either forced (microseconds of single
launches in a graph, with and without a gradient)."""
import ctypes

import pytest

# (rows, vocabulary, us with a gradient: a block per row, groups with a row in tensor memory; the same without a gradient)
MEASURED = [
    (3000, 8201, 39.4, 40.8, 30.8, 35.3), (3000, 9001, 45.5, 41.2, 35.6, 35.6), (620, 50257, 38.8, 42.5, 27.3, 30.9), (700, 50257, 39.6, 43.9, 28.2, 31.2),
    (920, 25001, 31.2, 32.6, 22.6, 25.6), (920, 50257, 54.0, 55.8, 36.9, 38.9), (1248, 20001, 33.8, 33.0, 25.2, 26.8), (1248, 15441, 28.1, 28.7, 21.0, 23.5),
    (1248, 50257, 68.5, 67.7, 46.9, 46.7), (1600, 25001, 51.6, 46.1, 37.1, 35.6), (800, 50257, 47.9, 45.6, 33.1, 32.0), (592, 50257, 33.6, 32.3, 24.0, 23.6),
    (592, 32003, 24.1, 23.0, 17.5, 18.0), (700, 32003, 28.4, 30.7, 21.5, 23.5), (722, 34425, 36.8, 32.6, 27.5, 24.9), (1251, 22492, 38.6, 35.5, 29.6, 28.9),
    (800, 25001, 27.5, 26.9, 20.2, 21.7), (3952, 8929, 55.9, 51.7, 44.2, 43.4), (2200, 40001, 98.8, 82.9, 67.2, 58.7), (620, 47321, 38.1, 39.9, 26.8, 29.2),
]


@pytest.fixture(scope="module")
def lib():
    from train_gpt_b200 import build, _lib
    build.build()
    return _lib.load()


def _in_groups(lib, rows, vocab):
    return bool(lib.tgh_softcap_ce_in_groups(ctypes.c_int64(rows), ctypes.c_int64(vocab)))


@pytest.mark.parametrize("rows,vocab,block_us,groups_us,block_fwd_us,groups_fwd_us", MEASURED)
def test_takes_the_faster_kernel_with_and_without_a_gradient(lib, rows, vocab, block_us, groups_us, block_fwd_us, groups_fwd_us):
    """(one kernel for both, so that a loss has the same bits either way: the gradient's time decides, and without one little is lost)"""
    if _in_groups(lib, rows, vocab):
        assert groups_us <= block_us and groups_fwd_us <= 1.075 * block_fwd_us
    else:
        assert block_us <= 1.01 * groups_us


def test_gpu_tests_reach_the_kernel_that_they_name(lib):
    from test_gpu_loss import LARGE_RAGGED, RAGGED
    assert all(_in_groups(lib, rows, vocab) for rows, vocab, _ in LARGE_RAGGED)
    assert not any(_in_groups(lib, rows, vocab) for rows, vocab, _ in RAGGED)
