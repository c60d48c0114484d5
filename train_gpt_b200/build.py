"""Build `libtrain_gpt_b200.so` (the C-ABI library, nvcc for sm_100a) and `_host.so` (the torch-facing host path,
g++ against torch's headers) in-tree.

    python -m train_gpt_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  Objects and libraries are written next to the
sources; a source newer than its library triggers a rebuild.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG_DIR), "include")
LIB_PATH = os.path.join(PKG_DIR, "libtrain_gpt_b200.so")
HOST_PATH = os.path.join(PKG_DIR, "_host.so")

SOURCES = ["runtime.cu", "quantize.cu", "rmsnorm.cu", "gemm_fp8.cu", "gemm_ring.cu", "gemm_skinny.cu", "selftest.cu", "loss.cu", "optim.cu"]

HOST_SOURCES = ["host.cpp", "step.cpp"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC")


def _stale(target: str, suffixes) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    deps = [os.path.join(d, f) for d in (CSRC, INCLUDE) for f in os.listdir(d) if f.endswith(suffixes)]
    return any(os.path.getmtime(d) > t for d in deps)


def _start_host():
    """Start compiling the host extension (it needs torch's headers and no GPU); returns what waits for it and links."""
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    inc = [*cpp_extension.include_paths(), os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include"),
           sysconfig.get_paths()["include"]]
    cmd = ["g++", "-fPIC", "-O2", "-std=c++17", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *[a for i in inc for a in ("-isystem", i)]]
    procs = []
    for src in HOST_SOURCES:
        obj = os.path.join(CSRC, src.replace(".cpp", "_host.o"))
        procs.append((src, obj, subprocess.Popen([*cmd, "-c", os.path.join(CSRC, src), "-o", obj], stdout=subprocess.PIPE,
                                                 stderr=subprocess.STDOUT, text=True)))

    def finish():
        outs = [(src, p.communicate()[0], p.returncode) for src, _, p in procs]
        for src, out, rc in outs:
            if rc != 0:
                raise RuntimeError(f"g++ failed on {src}:\n{out}")
        # (linked under another name and renamed when complete: another process never loads half a file)
        r = subprocess.run(["g++", "-shared", *[obj for _, obj, _ in procs], "-o", HOST_PATH + ".new",
                            "-L" + lib, "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda", "-ldl",
                            f"-Wl,-rpath,{lib}"], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link of _host.so failed:\n{r.stdout}")
        os.replace(HOST_PATH + ".new", HOST_PATH)

    return finish


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile what is missing or older than its sources; return the library's path."""
    finish_host = _start_host() if force or _stale(HOST_PATH, (".cpp", ".h")) else None
    if force or _stale(LIB_PATH, (".cu", ".cuh", ".h")):
        _build_lib(verbose)
    if finish_host is not None:
        finish_host()
    return LIB_PATH


def _build_lib(verbose: bool) -> None:
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(CSRC, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    log = []
    for src, p in procs:
        out, _ = p.communicate()
        log.append(f"== {src}\n{out}")
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
    link = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-lcudart"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    with open(os.path.join(CSRC, "build.log"), "w") as f:
        f.write("\n".join(log))
    if verbose:
        print("\n".join(log))


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
