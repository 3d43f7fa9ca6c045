"""Operations on pairs of double-floats (csrc/dfloat.h) give the bits of the single
operations: the arithmetic of the double-float integrator does not depend on which
components share an instruction.  Tolerance: none, every bit."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "etraj.jl_gb300", "csrc")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not found")
    out = str(tmp_path_factory.mktemp("pairs") / "libpairs.so")
    subprocess.run(["nvcc", "-std=c++17", "-O3", "--fmad=false", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-Xcompiler", "-fPIC", "-shared", "-I" + CSRC, os.path.join(HERE, "df_pair_probe.cu"), "-o", out],
                   check=True)
    return C.CDLL(out)


@pytest.mark.gpu
@pytest.mark.parametrize("span", [0, 3, 12])  # exponents of the values: -span .. span
def test_pairs_give_the_single_bits(probe, span):
    rng = np.random.default_rng(span)
    n = 4_000_000
    v = rng.uniform(-2, 2, n) * 2.0 ** rng.uniform(-span, span, n)
    v[::997] = 0.0
    v[1::997] = 1.0
    x = np.empty((n, 2), np.float32)
    x[:, 0] = v
    x[:, 1] = v - x[:, 0].astype(np.float64)
    counts = np.ones(9, np.uint64)
    rc = probe.df_pairs(x.ctypes.data_as(C.c_void_p), C.c_long(n), counts.ctypes.data_as(C.c_void_p))
    assert rc == 0
    assert not counts.any(), counts
