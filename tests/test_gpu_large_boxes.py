"""The FP64 walk where the rounding of its products passes the reference's ZERO
(an absolute 2.2e-12): boxes of side 100 and 1000, with rays through vertices and
along edges, whose signs there are noise.  Some rays end without an exit; each
ends as the oracle's, to the bit, and the mixed walk visits the same tets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = [1.0, 30.0, 100.0, 1000.0]
RECORD = 400


@pytest.fixture(scope="module")
def sd():
    import sdtfe_b200

    return sdtfe_b200


def trace_both(sd, oracle, pos4, tetra, L, xs, ys):
    budget = 2 * len(tetra) + 64
    want = oracle.trace(oracle.prepare(pos4, tetra, 1.0), xs, ys, 0.0, L, L / 24, 5, budget, RECORD)
    with sd.Mesh(pos4, tetra, 1.0) as m:
        out = [m.trace(sd.map_params(24, L, L, (L / 2,) * 3, 4, 0.0, 5, precision=p, max_visits=budget), xs, ys, 0.0, L,
                       L / 24, RECORD) for p in (sd.DTFE_FP64, sd.DTFE_MIXED)]
    (r64, c64, s64, v64), (r32, c32, s32, v32) = out
    assert np.array_equal(s64, want[2]) and np.array_equal(c64, want[1]) and np.array_equal(r64, want[0])
    ok = s64 == sd.RAY_OK
    assert np.array_equal(v64[ok], want[3][ok])
    assert np.array_equal(s32, s64) and np.array_equal(c32, c64) and np.array_equal(v32[ok], v64[ok])
    return s64


@pytest.mark.parametrize("L", SIDES)
def test_rays_through_the_particles(sd, oracle, L):
    rng = np.random.default_rng(11)
    pos4 = np.zeros((4000, 4))
    pos4[:, :3] = L * rng.random((4000, 3))
    status = trace_both(sd, oracle, pos4, sd.triangulate(pos4), L, pos4[:, 0].copy(), pos4[:, 1].copy())
    if L >= 100:  # the signs are noise there: the case is reached
        assert (status == sd.RAY_NO_EXIT).sum() > 100


@pytest.mark.parametrize("ss", [1, 2])
@pytest.mark.parametrize("L", SIDES)
def test_grids_and_maps_over_the_vertices(sd, oracle, L, ss):
    """Particles on the grid's own rays: every other ray runs through one."""
    G = 24 // ss
    rng = np.random.default_rng(12)
    ds = L / G / ss
    line = np.array([i * (L / G) + k * ds + ds / 2. for i in range(G) for k in range(ss)])
    on = np.stack(np.meshgrid(line, line), -1).reshape(-1, 2)[::2]
    xyz = np.concatenate([np.column_stack([on, L * rng.random(len(on))]), L * rng.random((500, 3))])
    pos4 = np.zeros((len(xyz), 4))
    pos4[:, :3] = xyz
    tetra = sd.triangulate(pos4)
    trace_both(sd, oracle, pos4, tetra, L, on[:, 0].copy(), on[:, 1].copy())
    centre, budget = (L / 2,) * 3, 2 * len(tetra) + 64
    prep = oracle.prepare(pos4, tetra, 1.0)
    want, _ = oracle.grid(prep, G, L, centre, ss, 4, budget)
    want_map = oracle.map(prep, G, L, L, centre, 3, 0.0, 9, budget)
    with sd.Mesh(pos4, tetra, 1.0) as m:
        got = m.grid(G, L, centre, ss, 4)
        st64 = m.last_stats()
        m.grid(G, L, centre, ss, 4, precision=sd.DTFE_MIXED)
        st32 = m.last_stats()
        got_map, _ = m.map(sd.map_params(G, L, L, centre, 3, 0.0, 9))
    assert np.array_equal(got, want)
    assert np.array_equal(got_map, want_map)
    assert (st64.visits, list(st64.status)) == (st32.visits, list(st32.status))
