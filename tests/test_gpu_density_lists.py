"""Vertex densities over tet lists of every length class (density.cuh): empty,
one tet, a full warp and one more, two, four warps of tets and one more.  The
sum runs from 0 in increasing tet order, so the densities equal a sequential
64-bit sum of the same volumes to the bit.  A tet out of range is refused and
nothing is written."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 130, 700]


def hubs():
    """A hub vertex per length, with that many tets to random other vertices, listed in mixed order."""
    rng = np.random.default_rng(5)
    n = len(LENGTHS) + 200
    pos4 = np.zeros((n, 4))
    pos4[:, :3] = rng.random((n, 3))
    rows = [[h, *(len(LENGTHS) + rng.choice(200, 3, replace=False))] for h, d in enumerate(LENGTHS) for _ in range(d)]
    rows = np.array([r[k:] + r[:k] for r, k in zip(rows, rng.integers(0, 4, len(rows)))])
    tetra = np.full((len(rows), 8), -1, np.int32)
    tetra[:, :4] = rows[rng.permutation(len(rows))]
    return pos4, tetra


def expected(pos4, tetra, mass):
    a, b, c, d = (pos4[tetra[:, k], :3] for k in range(4))
    a, b, c = a - d, b - d, c - d
    vol = np.abs((a[:, 0] * (b[:, 1] * c[:, 2] - b[:, 2] * c[:, 1]) + a[:, 1] * (b[:, 2] * c[:, 0] - b[:, 0] * c[:, 2])
                  + a[:, 2] * (b[:, 0] * c[:, 1] - b[:, 1] * c[:, 0])) / 6)
    total = np.zeros(len(pos4))
    for t, v in enumerate(vol):
        for k in tetra[t, :4]:
            total[k] += v
    with np.errstate(divide="ignore"):
        return float(np.float32(mass) * np.float32(4)) / total


def noalloc(pos4, tetra, mass):
    import torch

    import sdtfe_b200 as sd

    f = sd.lib().dtfe_density_noalloc
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_void_p,
                  ctypes.c_void_p]
    p, t = torch.from_numpy(pos4).cuda(), torch.from_numpy(tetra).cuda()
    rho = torch.full((len(pos4),), -7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return f(p.data_ptr(), len(pos4), t.data_ptr(), len(tetra), mass, rho.data_ptr(), None), rho.cpu().numpy()


@pytest.mark.parametrize("mass", [1.0, 0.3])
def test_densities_equal_a_sequential_sum(mass):
    import sdtfe_b200 as sd

    pos4, tetra = hubs()
    want = expected(pos4, tetra, mass)
    status, got = noalloc(pos4, tetra, mass)
    assert status == 0 and np.array_equal(got, want)
    with sd.Mesh(pos4, tetra, mass, flags=sd.MESH_LAZY) as m:
        assert np.array_equal(m.density(), want)
        assert list(m.adjacency()[:len(LENGTHS)]) == LENGTHS


@pytest.mark.parametrize("bad", [-1, 1 << 20])
def test_a_tet_out_of_range_writes_nothing(bad):
    pos4, tetra = hubs()
    tetra[len(tetra) // 2, 2] = bad
    status, got = noalloc(pos4, tetra, 1.0)
    assert status == 4 and np.all(got == -7.0)  # DTFE_ERR_MESH
    tetra[len(tetra) // 2, 2] = 0
    assert noalloc(pos4, tetra, 1.0)[0] == 0


def repeated():
    """hubs() with tets that list their hub twice, three and four times, some twice in a row of one
    list, in lists on both sides of 32, 64 and 128, and zero-filled padding rows (vertex 0 four times)."""
    pos4, tetra = hubs()
    rng = np.random.default_rng(6)
    for h, d in enumerate(LENGTHS):
        mine = np.flatnonzero((tetra[:, :4] == h).any(1))
        for t in rng.choice(mine, min(d, 5), replace=False):
            tetra[t, rng.choice(4, rng.integers(1, 5), replace=False)] = h
    pad = np.zeros((7, 8), np.int32)
    pad[:, 4:] = -1
    return pos4, np.concatenate([tetra[:50], pad, tetra[50:]])


@pytest.mark.parametrize("tets", [2, 7, 16, 19, 20, 37, 38, 39, 75, 77, 78, 300])
def test_one_list_of_repeated_tets(tets):
    """A hub that two of three of its tets list twice: lists on both sides of each length class."""
    rng = np.random.default_rng(tets)
    pos4 = np.zeros((60, 4))
    pos4[:, :3] = rng.random((60, 3))
    tetra = np.full((tets, 8), -1, np.int32)
    for row in tetra:
        row[:4] = rng.permutation([0, 0, *(1 + rng.choice(59, 2, replace=False))])
    # (tets with the hub twice have next to no volume: every third gets one)
    tetra[::3, 0] = np.where(tetra[::3, 0] == 0, 1 + rng.integers(59, size=len(tetra[::3])), tetra[::3, 0])
    status, got = noalloc(pos4, tetra, 1.0)
    assert status == 0 and np.array_equal(got, expected(pos4, tetra, 1.0))


def test_tets_that_list_a_vertex_several_times():
    import sdtfe_b200 as sd

    pos4, tetra = repeated()
    want = expected(pos4, tetra, 1.0)
    for _ in range(3):
        status, got = noalloc(pos4, tetra, 1.0)
        assert status == 0 and np.array_equal(got, want)
    with sd.Mesh(pos4, tetra, 1.0, flags=sd.MESH_LAZY) as m:
        assert np.array_equal(m.density(), want)
        assert np.array_equal(m.adjacency(), np.bincount(tetra[:, :4].ravel(), minlength=len(pos4)))
