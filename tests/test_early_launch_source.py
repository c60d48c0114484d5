"""Kernels that may start while the one before them on the stream still runs (programmatic dependent launch) have a rule that no run
on the GPU can be relied on to test: nothing that an earlier kernel writes is read before `grid_wait()`.  A plain load through a
`const __restrict__` parameter promises the compiler that the memory does not change while the kernel runs, so it may be moved above
the wait; such a pointer goes through `loads_below` after it.  Checked here by reading the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "train_gpt_b200", "csrc")


def _strip(text):
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", " ", text, flags=re.S))


def _balanced(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def _kernels():
    """(file, name, parameters, body) of every kernel that waits."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = _strip(open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__ void(?: __launch_bounds__\()?", text):
            at = m.end()
            if m.group().endswith("("):
                at = _balanced(text, at - 1, "()") + 1
            name = re.match(r"\s*(\w+)\s*\(", text[at:])
            open_at = at + name.end() - 1
            close_at = _balanced(text, open_at, "()")
            body_at = text.index("{", close_at)
            body = text[body_at:_balanced(text, body_at, "{}") + 1]
            if "grid_wait()" in body:
                out.append((f, name.group(1), text[open_at + 1:close_at], body))
    return out


KERNELS = _kernels()


def test_finds_the_kernels():
    names = {k[1] for k in KERNELS}
    assert {"rmsnorm_row_kernel", "skinny_reduce_kernel", "rmsnorm_dgamma_reduce_kernel", "splitk_reduce_kernel", "embed_kernel",
            "gemm_skinny_kernel", "gemm_fp8_blockscaled_kernel", "softcap_ce_kernel", "global_norm_kernel"} <= names


@pytest.mark.parametrize("f,name,params,body", KERNELS, ids=[k[1] for k in KERNELS])
def test_plain_loads_stay_below_the_wait(f, name, params, body):
    before, after = body.split("grid_wait()", 1)
    for p in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params):
        uses = [rf"\b{p}\s*\[", rf"\*\s*{p}\b(?!\s*[\w(])", rf"__ldc[gsav]\(\s*{p}\b", rf"_cast<const [^>]+>\({p}\b"]
        # a pointer made from it is as good as the parameter itself
        uses.append(rf"=\s*{p}\s*\+")
        plain = any(re.search(u, after) for u in uses)
        assert not any(re.search(u, before) for u in uses), (f, name, p)
        if plain:
            assert re.search(rf"\b{p} = loads_below\({p}\);", after), (f, name, p)


def test_no_load_takes_the_non_coherent_path():
    """`ld.global.nc` is for memory that nothing writes while the kernel runs.  A kernel launched early runs from before its input is
    written, and scratch that several kernels of a step reuse may still be held by that path with what it was."""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            text = _strip(open(os.path.join(CSRC, f)).read())
            assert "ld.global.nc" not in text and "__ldg(" not in text, f


def _bodies_with_start():
    """(file, name, body) of the device functions whose kernels pass the trigger and the wait in as `start`."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = _strip(open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__device__ __forceinline__ void (\w+)\(", text):
            close_at = _balanced(text, m.end() - 1, "()")
            if "START&&" in text[m.end():close_at]:
                body_at = text.index("{", close_at)
                out.append((f, m.group(1), text[body_at:_balanced(text, body_at, "{}") + 1]))
    return out


STARTED = _bodies_with_start()


def test_finds_the_bodies_behind_the_kernels():
    assert {b[1] for b in STARTED} == {"gemm_body", "ring_body"}
    for f, name, _, body in KERNELS:            # and a kernel that hands its wait on does nothing else before it
        if name in ("gemm_fp8_blockscaled_kernel", "gemm_two_kernel", "gemm_ring_kernel", "gemm_ring_two_kernel"):
            assert re.search(r"\[\] \{\s*grid_trigger\(\);\s*grid_wait\(\);\s*\}", body), name


@pytest.mark.parametrize("f,name,body", STARTED, ids=[b[1] for b in STARTED])
def test_bodies_touch_no_memory_before_their_start(f, name, body):
    """Scales, operands and results are read and written below `start()` only: no copy, no load through a pointer of the parameters."""
    assert body.count("start();") == 1
    before = body[:body.index("start();")]
    for access in (r"tma_load", r"tma_store", r"cp_async", r"cp\.async", r"\bld_\w+\(", r"__ldc[gsav]\(", r"ld\.global", r"\.sa\b", r"\.sb\b", r"\.d\b", r"\bpromote"):
        assert not re.search(access, before), (f, name, access)
