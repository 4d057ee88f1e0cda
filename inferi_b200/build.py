"""Builds libinferi_b200.so (sm_100a only) in-tree with nvcc, and the Python binding of the op launches.

The shared library is the product: a C-ABI (include/inferi_b200.h) with no torch or Python types in it, which needs neither to be built.  The binding
(csrc/binding.cpp) is what `ops.py` calls it through where there is one for the running interpreter and torch; without it calls go through ctypes.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libinferi_b200.so")
BINDING_PATH = os.path.join(PKG_DIR, "_binding" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))   # (another interpreter does not find it)
BINDING_SOURCES = [os.path.join(CSRC, "binding.cpp"), os.path.join(PKG_DIR, "..", "include", "inferi_b200.h"), os.path.abspath(__file__)]
SOURCES = ["api.cu", "gemv.cu", "gemv_stream.cu", "ops.cu", "attention.cu", "prefill.cu", "prefill_gemm.cu", "prefill_attention.cu", "llama.cu", "gguf.cu", "sampler.cu", "tokenizer.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; inferi_b200 needs the CUDA toolkit to build")


def _older(path: str, deps: list[str]) -> bool:
    return not os.path.exists(path) or any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def _stale() -> bool:
    return _older(LIB_PATH, [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f != "binding.cpp"] + BINDING_SOURCES[1:])


def binding_stamp() -> str:
    """The torch that a binding is for: it reads tensors through inline accessors, which another torch may lay out otherwise."""
    import torch

    return f"torch {torch.__version__} {torch.version.git_version}"


def _binding_command() -> list[str] | None:
    """How the binding is compiled: against this interpreter and its torch.  None without a torch, and with one that has no CUDA: no launch gets as far
    as the binding there."""
    try:
        import torch
    except ImportError:
        return None
    if torch.version.cuda is None:
        return None
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    includes = [f"{root}/include", f"{root}/include/torch/csrc/api/include", f"{cuda}/include", sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++20", "-shared", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
            f'-DIB_BINDING_STAMP="{binding_stamp()}"', *[f"-I{i}" for i in includes], BINDING_SOURCES[0], "-o", BINDING_PATH, f"-L{root}/lib", "-lc10", "-lc10_cuda",
            "-ltorch_cpu", "-ltorch_python", f"-Wl,-rpath,{root}/lib"]


def _binding_stale() -> bool:
    if _older(BINDING_PATH, BINDING_SOURCES):
        return True
    with open(BINDING_PATH, "rb") as f:
        return binding_stamp().encode() not in f.read()


def _start(cmd: list[str]) -> subprocess.Popen | None:
    try:
        return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    except OSError as e:   # no such compiler
        sys.stderr.write(f"{cmd[0]}: {e}\n")
        return None


def _finish_binding(p: subprocess.Popen | None, verbose: bool) -> None:
    """A binding that cannot be built is no error, and none is left behind that is not of these sources."""
    out = p.communicate()[0] if p else ""
    failed = p is None or p.returncode != 0
    if failed and os.path.exists(BINDING_PATH):
        os.remove(BINDING_PATH)
    if failed or verbose:
        sys.stderr.write(f"--- binding.cpp ---\n{out}\n")
    if failed:
        sys.stderr.write("the Python binding was not built; op launches go through ctypes\n")


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu of the package into libinferi_b200.so; returns its path.  And the binding, where there is a torch to compile it against."""
    command = _binding_command()
    wanted = command is not None and (force or _binding_stale())
    binding = _start(command) if wanted else None
    try:
        if force or _stale():
            _build_library(verbose)
    finally:
        if wanted:
            _finish_binding(binding, verbose)
    return LIB_PATH


def _build_library(verbose: bool) -> None:
    nvcc = _nvcc()
    objs = []
    build_dir = os.path.join(PKG_DIR, "build")
    os.makedirs(build_dir, exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = os.path.join(build_dir, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- nvcc {src} ---\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed; see the messages above")
    link = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-lcudart_static", "-lpthread", "-ldl", "-lrt"]
    subprocess.run(link, check=True)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
