"""Supersampled grids walked by sub-rays (grid_rays.cuh): the same cells, to
the bit in FP64, as the oracle's column after column, on sides and
supersamplings around the warp patches, onto a grid that holds values, and
with columns that leave the mesh or come back to a node they have passed."""
import numpy as np
import pytest

from conftest import MESH_SETS, golden_set

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sd():
    import sdtfe_b200

    return sdtfe_b200


@pytest.mark.parametrize("G,ss,box", [(1, 2, 0.5), (3, 3, 1.0), (4, 2, 0.9), (7, 5, 1.3), (17, 2, 1.0), (33, 3, 0.2)])
@pytest.mark.parametrize("name", MESH_SETS)
def test_subray_grid_equals_the_oracle(golden, sd, oracle, name, G, ss, box):
    s = golden_set(golden, name)
    prep = oracle.prepare(s["pos4"], s["tetra"], 1.0)
    # the oracle accumulates from zero: the grid's start value is one addend more
    want, _ = oracle.grid(prep, G, box, (0.5, 0.5, 0.5), ss, 4)
    with sd.Mesh(s["pos4"], s["tetra"], 1.0) as m:
        got = m.grid(G, box, (0.5, 0.5, 0.5), ss, 4)
        st64 = m.last_stats()
        mixed = m.grid(G, box, (0.5, 0.5, 0.5), ss, 4, precision=sd.DTFE_MIXED)
        st32 = m.last_stats()
        onto = m.grid(G, box, (0.5, 0.5, 0.5), ss, 4, out=np.full((G, G, G), 0.5))
    assert np.array_equal(got, want)
    assert np.all(np.abs(mixed - want) <= 1e-5 * np.abs(want))
    assert np.allclose(onto, want + 0.5, rtol=1e-13, atol=0)
    assert (st64.rays, st64.visits, list(st64.status)) == (st32.rays, st32.visits, list(st32.status))
    assert st64.rays == G * G and sum(st64.status) == G * G
