"""Builds libinferi_b200.so (sm_100a only) in-tree with nvcc, and the Python binding of the op launches.

The shared library is the product: a C-ABI (include/inferi_b200.h) with no torch or Python types in it.  `_binding.so` is what `ops.py` calls it
through where it can (csrc/binding.cpp).
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
BINDING_PATH = os.path.join(PKG_DIR, "_binding.so")
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


def _stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(PKG_DIR, "..", "include", "inferi_b200.h"), __file__]
    return any(os.path.getmtime(d) > t for d in deps) or not os.path.exists(BINDING_PATH)


def _binding_command() -> list[str] | None:
    """How the Python binding of the op launches is compiled (csrc/binding.cpp): against this interpreter and its torch.  None with a torch that has no
    CUDA: no launch gets as far as the binding there."""
    import torch

    if torch.version.cuda is None:
        return None
    root = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    includes = [f"{root}/include", f"{root}/include/torch/csrc/api/include", f"{cuda}/include", sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++20", "-shared", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
            *[f"-I{i}" for i in includes], os.path.join(CSRC, "binding.cpp"), "-o", BINDING_PATH, f"-L{root}/lib", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
            f"-Wl,-rpath,{root}/lib"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu of the package into libinferi_b200.so; returns its path."""
    if not force and not _stale():
        return LIB_PATH
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
    binding = _binding_command()
    if binding:
        procs.append(("binding.cpp", subprocess.Popen(binding, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {src} ---\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("the compiler failed; see the messages above")
    link = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-lcudart_static", "-lpthread", "-ldl", "-lrt"]
    subprocess.run(link, check=True)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
