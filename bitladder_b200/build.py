"""Builds ``libbitdecode.so`` (the C-ABI library) in-tree with nvcc for sm_100a.

Run as ``python -m bitladder_b200.build`` or call :func:`build`.  nvcc
cross-compiles without a GPU, so this works on a CPU-only host; the resulting
shared object sits beside this file and is what :mod:`bitladder_b200._lib` loads.
``_torch_calls.so`` beside it (g++, the headers of the installed torch) takes the operators' calls
on torch tensors to that library; without it they take interpreted code, so that where it cannot be
built the library still is.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
import warnings
from concurrent.futures import ThreadPoolExecutor

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(_HERE, "csrc")
BUILD_DIR = os.path.join(_HERE, "build")
LIB_PATH = os.path.join(_HERE, "libbitdecode.so")
CALLS_PATH = os.path.join(_HERE, "_torch_calls.so")
CALLS_SOURCE = os.path.join(CSRC, "bd_torch.cpp")
SOURCES = ["bd_pack.cu", "bd_decode.cu", "bd_decode_short.cu", "bd_combine.cu", "bd_exchange.cu", "bd_rope.cu", "bd_api.cu"]
HEADERS = ["bd_common.cuh", "bd_decode.cuh", "bd_pack.cuh", "bd_kernels.h", os.path.join("..", "..", "include", "bitdecode.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


# Per-file additions.  The decode kernel may use the approximate exp/log/division and
# flush-to-zero fp32 (its parity bound is 2e-3 and these act on softmax weights and the final
# normalisation; measured 0.8 us on a 63 us step).  The pack kernel must NOT: its quantizer is
# bit-exact IEEE arithmetic with explicit rounding intrinsics.
PER_FILE_FLAGS = {"bd_decode.cu": ["--use_fast_math"]}


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: cannot build libbitdecode.so")


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def calls_key() -> str:
    """What the extension's binary interface depends on: the installed torch and the interpreter."""
    import torch
    return f"torch {torch.__version__}, {sysconfig.get_config_var('SOABI')}"


def _calls_key_path() -> str:
    return os.path.join(BUILD_DIR, "torch_calls.key")


def _calls_stale(header: str) -> bool:
    if _stale(CALLS_PATH, [CALLS_SOURCE, os.path.abspath(__file__), header]) or not os.path.exists(_calls_key_path()):
        return True
    with open(_calls_key_path()) as f:
        return f.read() != calls_key()


def _build_calls() -> None:
    """The extension; a failure leaves none (an old one may have another layout of the argument blocks)."""
    for path in (CALLS_PATH, _calls_key_path()):
        if os.path.exists(path):
            os.remove(path)
    try:
        _run(_calls_command())
    except (ImportError, OSError, RuntimeError) as exc:
        warnings.warn(f"bitladder_b200._torch_calls is not built, calls on tensors cost 20 to 30 us more: {exc}")
        return
    with open(_calls_key_path(), "w") as f:
        f.write(calls_key())


def _calls_command():
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    return [os.environ.get("CXX") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DBD_BUILT_FOR="{calls_key()}"',
            *(f"-I{d}" for d in (os.path.join(root, "include"), os.path.join(cuda, "include"), sysconfig.get_paths()["include"])),
            CALLS_SOURCE, "-o", CALLS_PATH, f"-L{os.path.join(root, 'lib')}", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]


def _run(cmd) -> str:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("build failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return r.stdout + r.stderr


def build(force: bool = False, verbose: bool = False, extra_flags=()) -> str:
    """Compile every CUDA source and link the shared library; returns its path."""
    nvcc = _nvcc()
    os.makedirs(BUILD_DIR, exist_ok=True)
    hdrs = [os.path.normpath(os.path.join(CSRC, h)) for h in HEADERS]
    jobs = []
    objs = []
    for src in SOURCES:
        spath = os.path.join(CSRC, src)
        obj = os.path.join(BUILD_DIR, src.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [spath, os.path.abspath(__file__)] + hdrs):
            cmd = [nvcc, *NVCC_FLAGS, *PER_FILE_FLAGS.get(src, []), *extra_flags, "-c", spath, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    if jobs:
        with ThreadPoolExecutor(max_workers=min(4, len(jobs))) as ex:
            for out in ex.map(_run, jobs):
                if verbose and out:
                    print(out)
    if force or _stale(LIB_PATH, objs):
        _run([nvcc, "-shared", "-o", LIB_PATH, *objs, "-lcudart"])
    if force or _calls_stale(hdrs[-1]):
        _build_calls()
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
