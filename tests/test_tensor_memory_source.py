"""A kernel lets the kernels after it start early (`grid_trigger`) only once it has its tensor memory.  A dependent that reached an SM first
would allocate, wait for the kernel before it and never give the columns back that this one is still waiting for.  No run on
the GPU can be relied on to show it; checked here by reading the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "train_gpt_b200", "csrc")


def _bodies():
    """(file, name, body) of every function that allocates tensor memory, the wrappers of the instructions left out."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", " ", open(os.path.join(CSRC, f)).read(), flags=re.S))
        for m in re.finditer(r"^(?:__global__|__device__)[^;{]*?(\w+)\s*\((?=[^;{]*\{)", text, flags=re.M):
            at = text.index("{", m.end())
            end = re.compile(r"^}", flags=re.M).search(text, at).end()
            if "tmem_alloc(" in text[at:end] or "tcgen05.alloc" in text[at:end]:
                out.append((f, m.group(1), text[at:end]))
    return out


BODIES = _bodies()


def test_finds_the_kernels():
    assert {f for f, _, _ in BODIES} == {"gemm_fp8.cu", "gemm_ring.cu", "gemm_skinny.cu", "loss.cu", "selftest.cu"}


@pytest.mark.parametrize("f,body", [(f, b) for f, _, b in BODIES], ids=[f for f, _, _ in BODIES])
def test_dependents_start_after_the_allocation(f, body):
    allocated = max(m.end() for m in re.finditer(r"tmem_alloc\(|tcgen05\.alloc", body))
    met = body.index("__syncthreads();", allocated)                  # the allocating warp is through it when all threads are here
    triggers = [m.start() for m in re.finditer(r"grid_trigger\(\)|\bstart\(\)", body)]
    assert all(t > met for t in triggers), f
    assert triggers or f == "selftest.cu"
