"""The mixed walk's links between records (walk32.cuh): meshes where some or
all of them cannot be used, the smallest meshes, and the visit budget.  The
mixed walk must end like the FP64 walk: same tets, same order, same status.
Ray integrals within 1e-5 relative, the mixed path's bound, where chords join."""
import numpy as np
import pytest

from conftest import golden_set

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sd():
    import sdtfe_b200

    return sdtfe_b200


def same_walks(sd, pos4, tetra, xs, ys, max_visits=4000, values=True):
    with sd.Mesh(pos4, tetra, 1.0) as m:
        out = []
        for prec in (sd.DTFE_FP64, sd.DTFE_MIXED):
            p = sd.map_params(24, 1.0, 1.0, (0.5, 0.5, 0.5), 4, 0.0, 5, precision=prec,
                              max_visits=max_visits)
            out.append(m.trace(p, xs, ys, 0.0, 1.0, 1 / 24, 4000))
    (r64, c64, s64, v64), (r32, c32, s32, v32) = out
    assert np.array_equal(s32, s64) and np.array_equal(c32, c64)
    ok = s64 == sd.RAY_OK
    assert np.array_equal(v32[ok], v64[ok])
    if values:
        assert np.all(np.abs(r32 - r64)[ok] <= 1e-5 * np.abs(r64[ok]))
    return s64


@pytest.mark.parametrize("what", ["flipped", "flipped half", "swapped links"])
def test_meshes_with_unusable_links(golden, sd, what):
    """Tets listed with the other orientation (their faces are shared, but not
    with one orientation), and tets whose links are exchanged (a neighbour
    that does not hold the face)."""
    s = golden_set(golden, "clustered")
    tetra = s["tetra"].copy()
    rng = np.random.default_rng(3)
    pick = rng.random(len(tetra)) < (0.5 if what == "flipped half" else 0.03)
    if what == "swapped links":
        tetra[pick, 4], tetra[pick, 5] = s["tetra"][pick, 5], s["tetra"][pick, 4]
    else:
        for a, b in ((1, 2), (5, 6)):
            tetra[pick, a], tetra[pick, b] = s["tetra"][pick, b], s["tetra"][pick, a]
    # through exchanged links a ray crosses tets that do not touch: the walks
    # are the same, but no chord end is shared and the integrals mean nothing
    same_walks(sd, s["pos4"], tetra, s["trace_x"], s["trace_y"], values=what != "swapped links")


@pytest.mark.parametrize("n", [4, 5, 6, 9])
def test_smallest_meshes(sd, n):
    rng = np.random.default_rng(n)
    pos4 = np.zeros((n, 4))
    pos4[:, :3] = rng.random((n, 3)).astype(np.float32)
    tetra = sd.triangulate(pos4)
    xy = rng.random((500, 2))
    status = same_walks(sd, pos4, tetra, xy[:, 0], xy[:, 1])
    assert (status == sd.RAY_OK).any() and (status == sd.RAY_MISS).any()


@pytest.mark.parametrize("budget", [1, 2, 3, 17, 40])
def test_visit_budget(golden, sd, budget):
    s = golden_set(golden, "clustered")
    status = same_walks(sd, s["pos4"], s["tetra"], s["trace_x"], s["trace_y"], budget)
    assert (status == sd.RAY_BUDGET).any()


@pytest.mark.parametrize("what", ["flipped", "flipped half", "swapped links"])
def test_unusable_links_against_the_oracle(golden, sd, oracle, what):
    """The FP64 walk, which reads the same links as the mixed one: every ray ends as the oracle's, which
    reads none, to the bit."""
    s = golden_set(golden, "clustered")
    tetra = s["tetra"].copy()
    rng = np.random.default_rng(3)
    pick = rng.random(len(tetra)) < (0.5 if what == "flipped half" else 0.03)
    if what == "swapped links":
        tetra[pick, 4], tetra[pick, 5] = s["tetra"][pick, 5], s["tetra"][pick, 4]
    else:
        for a, b in ((1, 2), (5, 6)):
            tetra[pick, a], tetra[pick, b] = s["tetra"][pick, b], s["tetra"][pick, a]
    xy = rng.random((3000, 2))
    xs, ys = np.concatenate([s["trace_x"], xy[:, 0]]), np.concatenate([s["trace_y"], xy[:, 1]])
    want = oracle.trace(oracle.prepare(s["pos4"], tetra, 1.0), xs, ys, 0.0, 1.0, 1 / 24, 5, 4000, 4000)
    with sd.Mesh(s["pos4"], tetra, 1.0) as m:
        p = sd.map_params(24, 1.0, 1.0, (0.5, 0.5, 0.5), 4, 0.0, 5, max_visits=4000)
        got = m.trace(p, xs, ys, 0.0, 1.0, 1 / 24, 4000)
    ok = want[2] == sd.RAY_OK
    assert np.array_equal(got[2], want[2]) and np.array_equal(got[1], want[1]) and np.array_equal(got[0], want[0])
    assert np.array_equal(got[3][ok], want[3][ok])
