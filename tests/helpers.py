"""Shared helpers for the parity tests: torch tensors <-> the numpy oracle."""

import ctypes
import os
import subprocess

import numpy as np
import torch

from metile_b200 import build, synth
from oracle import affine as oracle


def triple_np(triple):
    """(packed, scales, biases) torch tensors -> numpy (uint32, float32, float32)."""
    packed, scales, biases = triple
    return (
        packed.detach().cpu().numpy().astype(np.uint32),
        synth.to_numpy_f32(scales),
        synth.to_numpy_f32(biases),
    )


def f32(tensor):
    return synth.to_numpy_f32(tensor)


def assert_within(actual, reference, rel=2e-3, what=""):
    """Every |y - y_ref| <= rel * max|y_ref| + one bf16 ulp (see oracle.affine.within_tolerance)."""
    ok, ratio = oracle.within_tolerance(f32(actual) if isinstance(actual, torch.Tensor) else actual,
                                        reference, rel)
    assert ok, f"{what}: worst error is {ratio:.2f}x the allowed bound (rel={rel:g})"
    return ratio


def assert_bit_equal(a, b, what=""):
    a16 = a.detach().cpu().contiguous().view(torch.uint16)
    b16 = b.detach().cpu().contiguous().view(torch.uint16)
    mismatches = int((a16 != b16).sum())
    assert mismatches == 0, f"{what}: {mismatches} of {a16.numel()} outputs differ bitwise"


def device_library(folder, source):
    """A shared library of kernels over the package's headers, compiled for the GPU."""
    path, library = os.path.join(folder, "kernels.cu"), os.path.join(folder, "kernels.so")
    with open(path, "w") as file:
        file.write(source)
    subprocess.run([build._nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-shared", "-Xcompiler", "-fPIC", "-I", build.CSRC, path, "-o", library], check=True)
    return ctypes.CDLL(library)


def host_program(folder, source):
    """Compile a program over the kernels' headers and run it HERE, without a GPU: the rows of integers it prints.
    For rules that the host and the device share, taken from where they stand."""
    path = os.path.join(folder, "program.cu")
    with open(path, "w") as file:
        file.write(source)
    binary = os.path.join(folder, "program")
    subprocess.run([build._nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", build.CSRC, path, "-o", binary], check=True)
    lines = subprocess.run([binary], check=True, capture_output=True, text=True).stdout.split("\n")
    return [tuple(int(word) for word in line.split()) for line in lines if line]
