"""Builds librustorch_attn.so (the C-ABI library) in-tree with nvcc for sm_100a, and _torch_binding.so, the
CPython extension through which the Python wrappers call it.

    python -m rustorch_b200.build [--force] [--verbose]

The same recipe is what a ``build.rs`` of the reference's ``rustorch-cuda`` crate would run:
one ``nvcc`` invocation over the ``csrc/*.cu`` translation units producing a shared (or static)
library that exports the symbols declared in ``include/rustorch_attn.h``.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "librustorch_attn.so")
BINDING_PATH = os.path.join(PKG_DIR, "_torch_binding.so")
BINDING_SOURCE = os.path.join(CSRC, "torch_binding.cpp")
SOURCES = ["api.cu", "decode.cu", "decode_tc.cu", "prefill_simt.cu", "prefill_tc.cu", "tc_selftest.cu", "decode_static.cu", "backward_simt.cu", "backward_tc.cu", "backward_tcgen05.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--use_fast_math=false",
    "-Xcompiler", "-fPIC",
    "-shared",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the attention library cannot be built")


def _sources() -> list[str]:
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def needs_build() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")] + [
        os.path.join(PKG_DIR, "..", "include", "rustorch_attn.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def _built_for() -> str:
    """What the extension is tied to besides its source: the interpreter, and the torch whose headers and libraries it uses."""
    import torch
    return f"{sys.implementation.cache_tag} {torch.__version__} abi{int(torch.compiled_with_cxx11_abi())}\n"


def binding_is_current() -> bool:
    """The extension is newer than its sources and was built for this interpreter and torch."""
    header = os.path.join(PKG_DIR, "..", "include", "rustorch_attn.h")
    stamp = BINDING_PATH + ".stamp"
    if not (os.path.exists(BINDING_PATH) and os.path.exists(stamp)):
        return False
    if os.path.getmtime(BINDING_PATH) <= max(os.path.getmtime(BINDING_SOURCE), os.path.getmtime(header)):
        return False
    with open(stamp) as f:
        return f.read() == _built_for()


def build_binding(force: bool = False) -> str:
    """g++ over torch_binding.cpp against torch's headers; linked to the C-ABI library next to it."""
    if not force and binding_is_current():
        return BINDING_PATH
    stamp = BINDING_PATH + ".stamp"
    if os.path.exists(stamp):  # a build that is cut short leaves no record
        os.remove(stamp)
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
    cmd += [x for d in includes for x in ("-isystem", d)] + ["-o", BINDING_PATH, BINDING_SOURCE]
    cmd += ["-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10",
            "-L" + PKG_DIR, "-l:" + os.path.basename(LIB_PATH), "-Wl,-rpath,$ORIGIN"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
        raise RuntimeError("g++ failed building _torch_binding.so")
    with open(stamp, "w") as f:
        f.write(_built_for())
    return BINDING_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        build_binding()
        return LIB_PATH
    cmd = [_nvcc()] + [f for f in NVCC_FLAGS if f != "--use_fast_math=false"]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB_PATH] + _sources() + ["-lcudart"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError("nvcc failed building librustorch_attn.so")
    build_binding(force)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
