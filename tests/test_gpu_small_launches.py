"""Small maps and grids walk fewer rays a warp (map_lanes32, grid_lanes32,
grid_lanes64).  Which lane walks a ray changes nothing of its result: maps must
equal, to the bit, those of a kernel variant that fills its warps, FP64 grids
the oracle's, and mixed grids the FP64 grids within the mixed path's 1e-5."""
import numpy as np
import pytest

from conftest import golden_set

pytestmark = pytest.mark.gpu

FULL_WARPS = 3  # a variant of 128 threads that always walks 32 rays a warp


@pytest.fixture(scope="module")
def sd():
    import sdtfe_b200

    return sdtfe_b200


@pytest.fixture(scope="module")
def mesh(golden, sd):
    s = golden_set(golden, "clustered")
    with sd.Mesh(s["pos4"], s["tetra"], 1.0) as m:
        yield m


# around 16,384, 24,576 and 32,768 rays, a pixel's samples around a block's room at 4 and
# 16 rays a warp, and sides that fill no tile
@pytest.mark.parametrize("side,samples", [(1, 1), (1, 300), (3, 16), (3, 17), (5, 64), (5, 65), (17, 33), (64, 4),
                                          (128, 1), (129, 1), (61, 5), (128, 4), (64, 6), (157, 1), (181, 1), (182, 1)])
def test_maps_equal_full_warps(sd, mesh, side, samples):
    p = sd.map_params(side, 1.0, 1.0, (0.5, 0.5, 0.5), samples, 0.0, 3, precision=sd.DTFE_MIXED)
    out = []
    for variant in (-1, FULL_WARPS):
        mesh.set_variant(variant)
        got, st = mesh.map(p)
        out.append((got, st.rays, st.visits, list(st.status)))
    mesh.set_variant(-1)
    assert out[0][1] == side * side * samples
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]


# around 8,192 columns or sub-rays (FP64), 18,944 columns, 26,936 sub-rays and
# 42,624 of either (mixed)
@pytest.mark.parametrize("G,ss", [(1, 1), (5, 1), (13, 3), (45, 2), (46, 2), (68, 2), (69, 2), (90, 1), (91, 1),
                                  (82, 2), (83, 2), (103, 2), (104, 2),
                                  (137, 1), (138, 1)])
def test_grids(golden, sd, oracle, mesh, G, ss):
    s = golden_set(golden, "clustered")
    got = mesh.grid(G, 1.0, (0.5, 0.5, 0.5), ss, 3)
    want, _ = oracle.grid(oracle.prepare(s["pos4"], s["tetra"], 1.0), G, 1.0, (0.5, 0.5, 0.5), ss, 3)
    assert np.array_equal(got, want)
    mixed = mesh.grid(G, 1.0, (0.5, 0.5, 0.5), ss, 3, precision=sd.DTFE_MIXED)
    assert np.all(np.abs(mixed - got) <= 1e-5 * np.abs(got))


# the last sides whose warps of 8 and of 16 lanes are all resident (grid_lanes32), and the next
@pytest.mark.parametrize("G,ss", [(136, 1), (137, 1), (192, 1), (193, 1), (76, 2), (77, 2), (108, 2), (109, 2)])
def test_mixed_grids_at_the_resident_lines(sd, mesh, G, ss):
    want = mesh.grid(G, 1.0, (0.5, 0.5, 0.5), ss, 3)
    st64 = mesh.last_stats()
    got = mesh.grid(G, 1.0, (0.5, 0.5, 0.5), ss, 3, precision=sd.DTFE_MIXED)
    st32 = mesh.last_stats()
    assert np.all(np.abs(got - want) <= 1e-5 * np.abs(want))
    assert (st64.rays, st64.visits, list(st64.status)) == (st32.rays, st32.visits, list(st32.status))


# maps on either side of the blocks that are all resident at six an SM (kResidentMap32), and large samples
@pytest.mark.parametrize("side,samples", [(182, 1), (320, 1), (337, 1), (150, 4), (180, 4), (6, 2000), (30, 128), (31, 128)])
def test_resident_maps_equal_full_warps(sd, mesh, side, samples):
    test_maps_equal_full_warps(sd, mesh, side, samples)
