"""reciprocal_near (walk64.cuh), compiled for the host: the correctly rounded
reciprocal of a sum, from that of a sum a few ulps away, for random mantissas
and those next to powers of two, over the exponents that products can have."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def reciprocals(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    out = str(tmp_path_factory.mktemp("rec") / "libreciprocal_host.so")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-shared", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-Xcompiler", "-fPIC,-ffp-contract=off", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "sdtfe_b200", "csrc"),
                    os.path.join(ROOT, "tests", "reciprocal_host.cu"), "-o", out], check=True)
    f = ctypes.CDLL(out).reciprocals
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    f.restype = None
    return f


@pytest.mark.parametrize("ulps", [-8, -3, -1, 0, 1, 3, 8])
@pytest.mark.parametrize("exponent", [-39, -3, 0, 7, 513])
def test_correctly_rounded(reciprocals, ulps, exponent):
    rng = np.random.default_rng(exponent + 1000 * ulps + 10 ** 6)
    mantissa = np.concatenate([rng.integers(0, 1 << 52, 200_000), np.arange(4096), (1 << 52) - 2 - np.arange(4096)])
    s = np.ldexp(1.0 + np.ldexp(mantissa.astype(np.float64), -52), exponent)
    s *= rng.choice([-1.0, 1.0], len(s))
    near = (s.view(np.int64) + ulps).view(np.float64)
    out = np.zeros_like(s)
    reciprocals(s.ctypes.data, near.ctypes.data, len(s), out.ctypes.data)
    assert np.array_equal(out, 1.0 / s)
