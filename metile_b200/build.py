"""In-tree build of libmetile_b200.so (nvcc, sm_100a) and of the torch binding _native.so (g++).

`python -m metile_b200.build [--force] [--verbose]`.  The shared objects are written into the package
(metile_b200/csrc/libmetile_b200.so, metile_b200/_native.so) so they travel with the tree; nothing is
installed into site-packages and there is no JIT cache.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUTPUT = os.path.join(CSRC, "libmetile_b200.so")
SOURCES = ("metile_b200.cu",)
HEADERS = ("common.cuh", "ptx.cuh", "affine_gemv.cuh", "affine_gemv_mma.cuh", "affine_umma.cuh", "affine_mlp_fused.cuh", "meeting_slots.h", "add_rmsnorm.cuh", "gather_rows.cuh", "attention_decode.cuh", "peer_reduce.cuh",
           "dense_rows.cuh", os.path.join("..", "..", "include", "metile_b200.h"))
BINDING_SOURCE = os.path.join(CSRC, "binding.cpp")
BINDING_OUTPUT = os.path.join(HERE, "_native.so")
BINDING_TORCH = os.path.join(CSRC, "build", "native.torch")  # the torch version it was compiled against


def _nvcc():
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found; the CUDA extension cannot be built")
    return found


def _older(output, inputs):
    if not os.path.exists(output):
        return True
    built = os.path.getmtime(output)
    return any(os.path.getmtime(path) > built for path in inputs if os.path.exists(path))


def is_stale():
    return _older(OUTPUT, [os.path.join(CSRC, name) for name in SOURCES + HEADERS])


def _torch_version():
    import torch

    return f"{torch.__version__} {sys.version_info[:2]}"


def binding_is_stale():
    if _older(BINDING_OUTPUT, [BINDING_SOURCE, os.path.join(CSRC, HEADERS[-1])]):
        return True
    try:
        with open(BINDING_TORCH) as file:
            return file.read() != _torch_version()
    except OSError:
        return True


def _build_binding():
    """The CPython module that takes torch tensors: compiled against the installed torch's headers, linked
    to libmetile_b200.so by a path relative to itself."""
    import torch
    from torch.utils import cpp_extension

    command = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for path in cpp_extension.include_paths() + [sysconfig.get_path("include"), os.path.join(os.path.dirname(
            os.path.dirname(_nvcc())), "include")]:
        command += ["-isystem", path]
    libraries = os.path.join(os.path.dirname(torch.__file__), "lib")
    command += [BINDING_SOURCE, OUTPUT, f"-L{libraries}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
                "-ltorch", "-ltorch_python", "-Wl,-rpath,$ORIGIN/csrc", "-o", BINDING_OUTPUT]
    subprocess.run(command, check=True)
    os.makedirs(os.path.dirname(BINDING_TORCH), exist_ok=True)
    with open(BINDING_TORCH, "w") as file:
        file.write(_torch_version())


def build(force=False, verbose=False):
    if force or is_stale():
        command = [
            _nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
            "-shared", "-Xcompiler", "-fPIC,-fno-gnu-unique", "--expt-relaxed-constexpr", "-Xlinker", "-soname=libmetile_b200.so",
        ]
        if verbose:
            command += ["-Xptxas", "-v"]
        command += [os.path.join(CSRC, name) for name in SOURCES]
        command += ["-o", OUTPUT]
        subprocess.run(command, check=True)
    if force or binding_is_stale():
        _build_binding()
    return OUTPUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
