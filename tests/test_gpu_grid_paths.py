"""The ways a grid takes (grid_rays.cuh, dense_columns64): sub-rays whose rows are
partly or not written, columns that come back to a node they have passed, and one
thread a column where the cells outnumber the tets a thousandfold or the rows would
not fit.  FP64 cells equal the oracle's to the bit; mixed cells are within 1e-5."""
import numpy as np
import pytest

from conftest import golden_set

pytestmark = pytest.mark.gpu

CENTRE = (0.5, 0.5, 0.5)


@pytest.fixture(scope="module")
def sd():
    import sdtfe_b200

    return sdtfe_b200


def same_grids(sd, oracle, pos4, tetra, G, box, ss, max_err=1e-5):
    budget = 2 * len(tetra) + 64
    want, status = oracle.grid(oracle.prepare(pos4, tetra, 1.0), G, box, CENTRE, ss, 4, budget)
    with sd.Mesh(pos4, tetra, 1.0) as m:
        got = m.grid(G, box, CENTRE, ss, 4)
        st64 = m.last_stats()
        mixed = m.grid(G, box, CENTRE, ss, 4, precision=sd.DTFE_MIXED)
        st32 = m.last_stats()
    assert np.array_equal(got, want)
    assert np.all(np.abs(mixed - want) <= max_err * np.abs(want))
    assert list(st64.status) == list(np.bincount(status.ravel(), minlength=len(st64.status)))
    assert (st64.rays, st64.visits, list(st64.status)) == (st32.rays, st32.visits, list(st32.status))
    return want


@pytest.mark.parametrize("G,ss,box", [(9, 2, 4.0), (30, 2, 2.5), (21, 3, 4.0), (11, 4, 3.0), (7, 5, 6.0), (5, 2, 40.0)])
def test_rows_partly_written(golden, sd, oracle, G, ss, box):
    s = golden_set(golden, "clustered")
    want = same_grids(sd, oracle, s["pos4"], s["tetra"], G, box, ss)
    assert (want == 0).mean() > 0.5


@pytest.mark.parametrize("G,ss", [(20, 2), (13, 3), (16, 4)])
def test_columns_that_come_back_to_a_node(golden, sd, oracle, G, ss):
    """A tet whose neighbour ahead is replaced by one that the ray has left: the rays through that
    face go round until the visit budget, and add the nodes between again and again."""
    s = golden_set(golden, "clustered")
    pos4, clean = s["pos4"], s["tetra"]
    ds = 1.0 / G / ss
    at = [(G // 2) / G + ds / 2.]
    _, crossed, _, visits = oracle.trace(oracle.prepare(pos4, clean, 1.0), at, at, 0.0, 1.0, 1 / G, 4, 1 << 20, 400)
    path = visits[0, :crossed[0]]
    k = 3 * crossed[0] // 4
    tetra = clean.copy()
    slot = 4 + int(np.flatnonzero(clean[path[k], 4:] == path[k + 1])[0])
    tetra[path[k], slot] = path[k // 3]
    plain, _ = oracle.grid(oracle.prepare(pos4, clean, 1.0), G, 1.0, CENTRE, ss, 4)
    want = same_grids(sd, oracle, pos4, tetra, G, 1.0, ss)
    assert np.max(want / np.where(plain > 0, plain, np.inf)) > 5


@pytest.mark.parametrize("G,ss", [(199, 2), (200, 2), (201, 3), (200, 1), (51, 16)])
def test_few_tets_and_many_cells(sd, oracle, G, ss):
    rng = np.random.default_rng(8)
    pos4 = np.zeros((40, 4))
    pos4[:, :3] = rng.random((40, 3)).astype(np.float32)
    same_grids(sd, oracle, pos4, sd.triangulate(pos4), G, 1.1, ss)
