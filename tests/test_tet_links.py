"""The FP64 walk's carried triangle (walk64.cuh, tet_links.cuh), compiled for
the host: a face's crossing computed from the carried order equals, to the
bit, the reference's expression for that face (face_z64), for every entry
face, rotation and exit; and link_rotation accepts exactly the rotations."""
import ctypes
import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def tl(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    out = str(tmp_path_factory.mktemp("tl") / "libtet_links_host.so")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-shared", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-Xcompiler", "-fPIC,-ffp-contract=off", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "sdtfe_b200", "csrc"),
                    os.path.join(ROOT, "tests", "tet_links_host.cu"), "-o", out], check=True)
    L = ctypes.CDLL(out)
    L.tl_crossings.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_double] + [ctypes.c_void_p] * 3
    L.tl_rotation.argtypes = [ctypes.c_void_p] * 2
    L.tl_exit_slot.argtypes = [ctypes.c_void_p]
    return L


@pytest.mark.parametrize("size", [1.0, 1e-3, 1e-6])
def test_crossings_equal_the_faces(tl, size):
    rng = np.random.default_rng(int(1 / size))
    for _ in range(300):
        v = 0.4 + size * rng.random((4, 3))
        o = 0.4 + size * rng.random(2)
        face, entry, leave = np.zeros(4), np.zeros((4, 3)), np.zeros((4, 3))
        tl.tl_crossings(v.ctypes.data, o.ctypes.data, rng.uniform(0.2, 2.0), face.ctypes.data, entry.ctypes.data,
                        leave.ctypes.data)
        for F, k in itertools.product(range(4), range(3)):
            assert entry[F, k] == face[F]
            assert leave[F, k] == face[tl.tl_exit_face(F, k)]


def test_link_rotation(tl):
    w = np.array([7, 3, 9], np.int32)
    for p in itertools.permutations(range(3)):
        u = np.ascontiguousarray(w[list(p)])
        r = tl.tl_rotation(u.ctypes.data, w.ctypes.data)
        want = [k for k in range(3) if all(u[s] == w[(s + k) % 3] for s in range(3))]
        assert r == (want[0] if want else -1)
    other = np.array([7, 3, 8], np.int32)
    assert tl.tl_rotation(other.ctypes.data, w.ctypes.data) == -1


def test_exit_slot_for_every_combination_of_signs(tl):
    """The slot k with a_{k+1} < 0 < a_{k+2}; none when the three products, rounded, have one sign."""
    for signs in itertools.product((-1.0, 1.0), repeat=3):
        a = np.array(signs) * [1e-11, 3.0, 1e5]
        want = [k for k in range(3) if a[(k + 1) % 3] < 0 < a[(k + 2) % 3]]
        assert tl.tl_exit_slot(a.ctypes.data) == (want[0] if want else -1)
