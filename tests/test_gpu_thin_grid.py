"""Grids of one or two cells in a direction: a domain narrower than the
margins the cell grid adds around it.  The lists, the PPE matrix and its
right-hand side are the oracle's bit for bit and the pressure its within 1e-8,
with the multilevel and the IC(0) preconditioner.
"""
import ctypes as C

import numpy as np
import pytest

from mps_b200 import config as CF
from mps_b200 import types as T
from mps_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _column(dim, axis, cells):
    """A column of fluid on a wall inside a grid of `cells` cells along `axis`."""
    l0 = 0.02
    wl = (W.small_dambreak3d if dim == 3 else W.small_dambreak2d)(l0=l0, seed=5)
    cfg = wl.config()
    re = CF.neighbor_radius(cfg)
    k = [int(0.999 * cells * re / l0) if d == axis else 9 for d in range(dim)]
    up = (axis + 1) % dim
    k[up] = 14
    idx = np.stack(np.meshgrid(*[np.arange(m) for m in k], indexing="ij"), -1).reshape(-1, dim)
    pos = idx * l0
    pos[:, axis] += -4.0 * re + 0.25 * (cells * re - (k[axis] - 1) * l0)
    rng = np.random.default_rng(7)
    pos += rng.uniform(-0.01 * l0, 0.01 * l0, size=pos.shape)
    cfg.domain_min[axis] = 0.0
    cfg.domain_max[axis] = (cells - 2 - 8) * re + (0.5 if cells == 2 else -0.5) * re
    for d in range(dim):
        if d != axis:
            cfg.domain_min[d], cfg.domain_max[d] = 0.0, k[d] * l0
    types = np.where(idx[:, up] < 2, T.WALL, T.FLUID).astype(np.int32)
    return cfg, re, T.HostParticles(dim, pos, rng.normal(0.0, 0.05, size=pos.shape), types)


@pytest.mark.parametrize("sweep", ["3", "0"])
@pytest.mark.parametrize("dim,axis,cells", [(2, 0, 1), (2, 0, 2), (2, 1, 2), (3, 0, 1), (3, 0, 2), (3, 1, 1),
                                            (3, 1, 2), (3, 2, 1)])
def test_thin_grid_matches_the_oracle(dim, axis, cells, sweep, monkeypatch):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mps_b200.session import Session
    from oracle.pyoracle import Oracle
    monkeypatch.setenv("MPS_SWEEP", sweep)
    cfg, re, hp = _column(dim, axis, cells)
    orc = Oracle(dim)
    orc.initial_params(hp, cfg)
    nl = T.HostNeighborList(hp.n, cfg.max_neighbors)
    cl = orc.cell_list(hp.n, re, cfg)
    assert (cl.nx, cl.ny, getattr(cl, "nz", 0))[axis] == cells
    assert orc.search(nl, hp, cl, re) == 0
    orc.lib.oracle_number_density(C.byref(hp.ps), C.byref(nl.nl), C.byref(cfg))
    orc.lib.oracle_judge_free_surface(C.byref(hp.ps), cfg.surface_threshold)
    eq, rp, ci, va, b = orc.assemble(hp, nl, cfg)
    assert len(rp) > 10 and np.abs(b).max() > 0.0
    ho = hp.copy()
    assert orc.lib.oracle_solve_pressure(C.byref(ho.ps), C.byref(nl.nl), C.byref(cfg)) > 0
    m = cfg.max_neighbors
    with Session(cfg, dim, hp.n) as s:
        s.upload(hp)
        s.set_initial_params(hp.ps.n0, hp.ps.lambda_, hp.ps.n0_count)
        s.run_stage("solve_pressure", nl.neighbors[: hp.n * m], nl.count[: hp.n], m)
        geq, grp, gci, gva, gb = s.ppe()
        g = s.download()
        assert s.metrics()["converged"] == 1
    for x, y in ((geq, eq), (grp, rp), (gci, ci), (gva, va), (gb, b)):
        assert np.array_equal(x, y)
    p = ho.view["pressure"]
    assert np.linalg.norm(g["pressure"] - p) <= 1e-8 * np.linalg.norm(p)
