"""The neighbour lists built by a thread per particle (MPS_NBR_LANES=0, the
form of 60,000 particles and more) and the walk over the cells of a session
whose capacity leaves no room for lists: against the oracle as the lists by
eight lanes are, and a step bit for bit the default's.
"""
import numpy as np
import pytest

from mps_b200 import types as T
from mps_b200 import workloads as W

import test_gpu_lists as lists

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "pressure", "n", "type", "on_surface")


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("doubled", [False, True])
def test_thread_per_particle_matches_the_oracle(dim, doubled, monkeypatch):
    monkeypatch.setenv("MPS_NBR_LANES", "0")
    lists.test_lists_and_step_match_the_oracle(dim, doubled)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim", [2, 3])
def test_no_room_for_lists(dim, precision):
    """The lists of the capacity would take more than 24 GB: every operator
    walks the cells, and nothing of that size is allocated."""
    torch = _cuda()
    from mps_b200.session import start
    # 3-D: 592 neighbours at rest, 4 bytes each with room for 1.4 times as many; 2-D: 1,257
    wl = W.small_dambreak3d(l0=0.03, seed=23, influence_ratio_lap="5.2") if dim == 3 else \
        W.small_dambreak2d(l0=0.02, seed=23, influence_ratio_lap="20.0", influence_ratio_n="2.1")
    wl.params["max_neighbors"] = "2000"
    got = []
    for capacity in (None, 8_000_000 if dim == 3 else 4_000_000):
        hp = T.HostParticles(dim, wl.pos, wl.vel, wl.types)
        torch.cuda.synchronize()
        with start(wl.config(), dim, hp, capacity=capacity, precision=precision) as s:
            s.neighbor_search()
            before = torch.cuda.mem_get_info()[0]
            nb, cnt = s.neighbor_list(2000)
            s.step(2)
            used = before - torch.cuda.mem_get_info()[0]
            got.append((s.download(), nb, cnt, s.metrics()["total_iterations"]))
        assert used < (4 << 30)
    (a, nb, cnt, it), (b, nb2, cnt2, it2) = got
    assert np.array_equal(cnt, cnt2) and it == it2
    used = np.arange(2000)[None, :] < cnt[:, None]
    assert np.array_equal(nb.reshape(-1, 2000)[used], nb2.reshape(-1, 2000)[used])
    for f in FIELDS:
        assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("dim", [2, 3])
def test_matrix_of_rows_beyond_the_lists(dim):
    """Rows with more neighbours than a list holds are assembled from the cells,
    with run starts of their own: the matrix is the oracle's bit for bit, in
    both precision forms."""
    _cuda()
    import ctypes as C
    from mps_b200 import config as CF
    from mps_b200.session import Session
    from oracle.pyoracle import Oracle
    wl = lists._workload(dim, True)
    cfg = wl.config()
    orc = Oracle(dim)
    hp = T.HostParticles(dim, wl.pos, wl.vel, wl.types)
    orc.initial_params(hp, cfg)
    hp.ps.n0 *= 0.6   # fluid of twice the lattice's density: inside, not on the surface
    re = CF.neighbor_radius(cfg)
    m = cfg.max_neighbors
    nl = T.HostNeighborList(hp.n, m)
    cl = orc.cell_list(hp.n, re, cfg)
    assert orc.search(nl, hp, cl, re) == 0
    orc.lib.oracle_number_density(C.byref(hp.ps), C.byref(nl.nl), C.byref(cfg))
    orc.lib.oracle_judge_free_surface(C.byref(hp.ps), cfg.surface_threshold)
    want = orc.assemble(hp, nl, cfg)
    q = re / cfg.particle_distance
    k = np.arange(-4, 5)
    g = np.stack(np.meshgrid(*[k] * dim), -1).reshape(-1, dim)
    room = (int(1.4 * np.sum((g ** 2).sum(-1) < q * q)) + 15) & ~7
    unknown = want[0] >= 0
    assert (nl.count[: hp.n][unknown] > room).sum() > 100 and (nl.count[: hp.n][unknown] <= room).sum() > 100
    for precision in (0, 1):
        with Session(cfg, dim, hp.n, precision=precision) as s:
            s.upload(hp)
            s.set_initial_params(hp.ps.n0, hp.ps.lambda_, hp.ps.n0_count)
            s.run_stage("solve_pressure", nl.neighbors[: hp.n * m], nl.count[: hp.n], m)
            got = s.ppe()
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
