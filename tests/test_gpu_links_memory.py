"""The links between walk records (tet_links.cuh): one copy a mesh, shared by its
axes and both precisions, and none where a serving budget has no room for them beside
an FP64 request, which is then served by general steps alone.  Every map is the same
to the bit, as the mesh makes it by itself."""
import numpy as np
import pytest

from conftest import golden_set

pytestmark = pytest.mark.gpu

REC64, REC32, LINKS = 160, 128, 192  # bytes a tet


@pytest.fixture(scope="module")
def sd():
    import sdtfe_b200

    return sdtfe_b200


def params(sd, axis, precision, seed=3):
    return sd.map_params(48, 1.0, 1.0, (0.5, 0.5, 0.5), 4, 0.0, seed, axis=axis, precision=precision)


def test_one_copy_for_all_axes(golden, sd):
    s = golden_set(golden, "clustered")
    nt = len(s["tetra"])
    with sd.Mesh(s["pos4"], s["tetra"], 1.0, flags=sd.MESH_LAZY) as m:
        held = []
        for axis in range(3):
            m.hull(axis)
        for axis, precision in [(0, sd.DTFE_FP64), (1, sd.DTFE_FP64), (2, sd.DTFE_FP64), (1, sd.DTFE_MIXED)]:
            before = m.info().device_bytes
            m.map(params(sd, axis, precision))
            held.append((m.info().device_bytes - before) / nt)
    assert held == [REC64 + LINKS, REC64, REC64, REC32]


# bytes a tet beside one map: what FP64 needs without links, what mixed needs, both with links
@pytest.mark.parametrize("room", [REC64, REC32 + LINKS, REC64 + LINKS])
@pytest.mark.parametrize("held", [False, True])
def test_requests_under_a_budget(golden, sd, room, held):
    s = golden_set(golden, "clustered")
    nt = len(s["tetra"])
    asked = [(0, sd.DTFE_FP64), (1, sd.DTFE_FP64), (1, sd.DTFE_FP64)]
    if room >= REC32 + LINKS:
        asked += [(2, sd.DTFE_MIXED), (0, sd.DTFE_FP64), (1, sd.DTFE_MIXED), (2, sd.DTFE_MIXED)]
    with sd.Mesh(s["pos4"], s["tetra"], 1.0) as alone:
        want = [alone.map(params(sd, a, p))[0] for a, p in asked]
    budget = nt * room + 8 * 48 * 48
    # held: the mesh comes with records and links
    with sd.Mesh(s["pos4"], s["tetra"], 1.0, flags=0 if held else sd.MESH_LAZY) as m:
        assert m.info().fp32_exact
        with sd.Server(device_budget=budget) as srv:
            mid = srv.add_mesh(m)
            for (axis, precision), w in zip(asked, want):
                assert np.array_equal(srv.wait(srv.submit(mid, params(sd, axis, precision)))[0], w)
            st = srv.stats()
            assert st.peak <= budget and st.completed == len(asked)
            too_large = int(np.ceil(np.sqrt((budget - nt * REC64 + 1) / 8.0)))
            for p in [sd.map_params(too_large, 1.0, 1.0, (0.5, 0.5, 0.5), 1, 0.0, 1, axis=1)] + (
                    [params(sd, 1, sd.DTFE_MIXED)] if room < REC32 + LINKS else []):
                with pytest.raises(sd.DTFEError) as e:
                    srv.wait(srv.submit(mid, p))
                assert e.value.status == sd.ERR_ADMISSION
        # the mesh serves its owner as before
        for (axis, precision), w in zip(asked, want):
            assert np.array_equal(m.map(params(sd, axis, precision))[0], w)


def test_served_without_links_when_the_device_is_full(sd):
    """FP64 records without links, as the device has room for the records alone; a
    request over them that a server's budget has links for is served all the same."""
    import torch

    from sdtfe_b200 import workloads

    pos4, _ = workloads.clustered_box(n=200000, seed=7, n_clusters=6, r_max=0.05)
    tetra = sd.triangulate(pos4)
    nt, part = len(tetra), 64 << 20
    p = params(sd, 0, sd.DTFE_FP64)
    assert nt * LINKS > 3 * part  # more than is left beside the records
    with sd.Mesh(pos4, tetra, 1.0) as alone, sd.Server() as srv:
        want = alone.map(p)[0]
        assert np.array_equal(srv.wait(srv.submit(srv.add_mesh(alone), p))[0], want)
    with sd.Mesh(pos4, tetra, 1.0, flags=sd.MESH_LAZY) as m:
        for axis in range(3):
            m.hull(axis)
        sd.trim_memory()
        before, taken = m.info().device_bytes, []
        try:
            while torch.cuda.mem_get_info()[0] > nt * REC64 + 3 * part:
                taken.append(torch.empty(part, dtype=torch.uint8, device="cuda"))
            assert np.array_equal(m.map(p)[0], want)
            assert m.info().device_bytes == before + nt * REC64
            with sd.Server(device_budget=nt * (REC64 + LINKS) + part) as srv:
                assert np.array_equal(srv.wait(srv.submit(srv.add_mesh(m), p))[0], want)
            assert m.info().device_bytes == before + nt * REC64
        finally:
            taken.clear()
            torch.cuda.empty_cache()
        with sd.Server() as srv:  # room again: with its links
            assert np.array_equal(srv.wait(srv.submit(srv.add_mesh(m), p))[0], want)
