"""The compact neighbour lists of the device-resident step against the oracle.

The lists have room for 1.4 times the neighbours of the rest lattice; a
particle with more walks the cells instead, inside the same kernels.  The
fluid here is doubled by a second lattice inside the first, so that its
particles exceed the room and the walls' do not, at particle counts that leave
the last slice of 32 partly filled; the plain lattice stays below it.  Lists,
densities, flags and types come out bit for bit, pressures within 1e-8.
"""
import numpy as np
import pytest

from mps_b200 import config as CF
from mps_b200 import types as T
from mps_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _rel(a, b):
    nb = np.linalg.norm(b)
    return np.linalg.norm(a - b) / (nb if nb > 0 else 1.0)


def _workload(dim, doubled):
    l0 = 0.02 if dim == 3 else 0.0125
    wl = (W.small_dambreak3d if dim == 3 else W.small_dambreak2d)(l0=l0, seed=11)
    if doubled:
        f = wl.types == T.FLUID
        extra = wl.pos[f] + 0.45 * l0
        wl.pos = np.concatenate([wl.pos, extra])
        wl.vel = np.concatenate([wl.vel, np.zeros_like(extra)])
        wl.types = np.concatenate([wl.types, np.full(len(extra), T.FLUID, np.int32)])
    return wl


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("doubled", [False, True])
def test_lists_and_step_match_the_oracle(dim, doubled):
    _cuda()
    from mps_b200.session import Session
    from oracle.pyoracle import Oracle
    wl = _workload(dim, doubled)
    cfg = wl.config()
    orc = Oracle(dim)
    hp = T.HostParticles(dim, wl.pos, wl.vel, wl.types)
    orc.initial_params(hp, cfg)
    re = CF.neighbor_radius(cfg)
    m = cfg.max_neighbors
    nl = T.HostNeighborList(hp.n, m)
    cl = orc.cell_list(hp.n, re, cfg)
    assert orc.search(nl, hp, cl, re) == 0
    q = re / wl.config().particle_distance
    k = np.arange(-4, 5)
    g = np.stack(np.meshgrid(*[k] * dim), -1).reshape(-1, dim)
    room = (int(1.4 * np.sum((g ** 2).sum(-1) < q * q)) + 15) & ~7
    assert (nl.count[: hp.n].max() > room) == doubled and hp.n % 32 != 0
    with Session(cfg, dim, hp.n) as s:
        s.upload(hp)
        s.set_initial_params(hp.ps.n0, hp.ps.lambda_, hp.ps.n0_count)
        s.neighbor_search()
        nb, cnt = s.neighbor_list(m)
        s.step(1)
        out = s.download()
    assert np.array_equal(cnt, nl.count[: hp.n])
    for i in range(hp.n):
        assert np.array_equal(nb[i * m: i * m + cnt[i]], nl.neighbors[i * m: i * m + cnt[i]]), i
    assert orc.step(hp, nl, cl, cfg) == 0
    o = hp.view
    for f in ("n", "on_surface", "type"):
        assert np.array_equal(out[f], o[f]), f
    assert _rel(out["pressure"], o["pressure"]) < 1e-8
    assert _rel(out["vel"], o["vel"]) < 1e-10
    assert _rel(out["pos"], o["pos"]) < 1e-14
