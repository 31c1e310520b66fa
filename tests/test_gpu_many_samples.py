"""FP64 maps on either side of the block sizes that the samples a pixel choose
(map_block64 and kFewPixels64 in walk.cu), alone, in batches whose maps need several
launches, and served: every map equals the oracle's to the bit."""
import numpy as np
import pytest

from conftest import golden_set

pytestmark = pytest.mark.gpu

CENTRE = (0.5, 0.5, 0.5)


@pytest.fixture(scope="module")
def sd():
    import sdtfe_b200

    return sdtfe_b200


@pytest.fixture(scope="module")
def mesh(golden, sd, oracle):
    s = golden_set(golden, "clustered")
    with sd.Mesh(s["pos4"], s["tetra"], 1.0) as m:
        yield m, oracle.prepare(s["pos4"], s["tetra"], 1.0)


@pytest.mark.parametrize("G,S", [(5, 64), (5, 65), (3, 129), (4, 257), (50, 65), (51, 65), (51, 100), (52, 128), (51, 129),
                                 (3, 4096), (3, 4097), (52, 300), (2, 16384)])
def test_map(sd, oracle, mesh, G, S):
    m, prep = mesh
    p = sd.map_params(G, 1.0, 1.0, CENTRE, S, 0.0, 17)
    want, rho, crossed, _ = oracle.map(prep, G, 1.0, 1.0, CENTRE, S, 0.0, 17, per_ray=True)
    got, st = m.map(p)
    assert np.array_equal(got, want) and st.rays == G * G * S
    got, _, ray_rho, ray_crossed, _ = m.map(p, per_ray=True)
    assert np.array_equal(got, want) and np.array_equal(ray_rho, rho) and np.array_equal(ray_crossed, crossed)


JOBS = [(9, 4), (7, 65), (2, 5000), (6, 64), (5, 300), (12, 16), (2, 4097), (3, 4096)]


@pytest.mark.parametrize("jobs", [JOBS, JOBS[:2], [JOBS[2]], [(9, 4), (2, 5000)], [(7, 65)]])
@pytest.mark.parametrize("graph", [False, True])
def test_batch(sd, oracle, mesh, jobs, graph):
    import torch

    m, prep = mesh
    maps = [torch.zeros((G, G), dtype=torch.float64, device="cuda") for G, _ in jobs]
    ps = [sd.map_params(G, 1.0, 1.0, CENTRE, S, 0.0, 30 + k) for k, (G, S) in enumerate(jobs)]
    torch.cuda.synchronize()
    b = sd.Batch([(m, p, d.data_ptr()) for p, d in zip(ps, maps)],
                 flags=sd.BATCH_ZERO_MAPS | (sd.BATCH_GRAPH if graph else 0))
    for _ in range(2):
        b.launch()
        b.sync()
        for k, (G, S) in enumerate(jobs):
            assert np.array_equal(maps[k].cpu().numpy(), oracle.map(prep, G, 1.0, 1.0, CENTRE, S, 0.0, 30 + k))
            assert b.stats()[k].rays == G * G * S
    b.close()


def test_served(sd, oracle, mesh):
    m, prep = mesh
    with sd.Server(quantum_rays=1 << 10) as srv:
        mid = srv.add_mesh(m)
        rids = [srv.submit(mid, sd.map_params(G, 1.0, 1.0, CENTRE, S, 0.0, 30 + k)) for k, (G, S) in enumerate(JOBS)]
        for k, (rid, (G, S)) in enumerate(zip(rids, JOBS)):
            assert np.array_equal(srv.wait(rid)[0], oracle.map(prep, G, 1.0, 1.0, CENTRE, S, 0.0, 30 + k))
