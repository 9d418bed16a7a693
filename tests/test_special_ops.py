"""The branch-free square roots, reciprocals and divisions that the step kernels' bit-identity rests on (itr_device.cuh),
against CUDA's IEEE-rounded operations: every 32-bit operand of the ranges of rcp2 and sqrt2 (and their scalar forms), a
dense seeded sample with the edges of Fast::div, div_rn and div_by_f32, and the twice-rounded paired product and sum.
"""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NAMES = ["rcp2", "Fast::rcp", "sqrt2", "Fast::sqrt", "Fast::div", "Fast::div below the normal range", "div_rn", "div_by_f32", "mul2 and add2"]


def build(out):
    """With the library's flags: no contraction, IEEE division and square root, no flush to zero."""
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false", "-prec-div=true", "-prec-sqrt=true",
                    "-ftz=false", "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(ROOT, "inverse-terrain-engine_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-o", str(out), os.path.join(ROOT, "tests", "special_ops.cu"), "-lcudart"], check=True)
    return str(out)


def test_special_ops_source_builds(tmp_path):
    assert os.path.getsize(build(tmp_path / "special_ops.so")) > 0


@pytest.mark.gpu
def test_branch_free_operations_are_the_ieee_ones(tmp_path):
    lib = C.CDLL(build(tmp_path / "special_ops.so"))
    n = (C.c_ulonglong * len(NAMES))()
    assert lib.special_ops(n, C.c_ulonglong(1 << 30)) == 0
    assert dict(zip(NAMES, n)) == dict.fromkeys(NAMES, 0)
