"""Plain CG (solver_type 0, the configuration's default) on the GPU.

A step against the oracle's CG in 3-D and 2-D and both precision forms
(pressure 1e-8, velocity 1e-10, position 1e-14 relative L2, as for a
preconditioned step), and the mixed form's product from packed words: one
launch fewer than from the separate arrays (MPS_PACK=0), which a conversion
makes first, and the same bits.  Its reliable updates come every hundredfold
fall of the residual, every ten thousandfold in the multilevel form.
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
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _workload(dim):
    return (W.small_dambreak3d if dim == 3 else W.small_dambreak2d)(l0=0.02, seed=17, solver_type=0)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dim", [2, 3])
def test_step_matches_the_oracle(dim, precision):
    _cuda()
    from mps_b200.session import start
    from oracle.pyoracle import Oracle
    wl = _workload(dim)
    cfg = wl.config()
    assert cfg.solver_type == 0
    with start(cfg, dim, T.HostParticles(dim, wl.pos, wl.vel, wl.types), precision=precision) as s:
        s.step(1)
        g, m = s.download(), s.metrics()
    orc = Oracle(dim)
    hp = T.HostParticles(dim, wl.pos, wl.vel, wl.types)
    orc.initial_params(hp, cfg)
    re = CF.neighbor_radius(cfg)
    nl = T.HostNeighborList(hp.n, cfg.max_neighbors)
    cl = orc.cell_list(hp.n, re, cfg)
    assert orc.search(nl, hp, cl, re) == 0
    assert orc.step(hp, nl, cl, cfg) == 0
    assert m["converged"] == 1 and m["ppe_iterations"] > 10
    o = hp.view
    for f in ("n", "on_surface", "type"):
        assert np.array_equal(g[f], o[f]), f
    assert _rel(g["pressure"], o["pressure"]) < 1e-8
    assert _rel(g["vel"], o["vel"]) < 1e-10
    assert _rel(g["pos"], o["pos"]) < 1e-14


@pytest.mark.parametrize("dim", [2, 3])
def test_mixed_product_reads_packed_words(dim, monkeypatch):
    _cuda()
    from mps_b200.session import start
    wl = _workload(dim)
    out, launches, iters = [], [], []
    for pack in ("1", "0"):
        monkeypatch.setenv("MPS_PACK", pack)
        with start(wl.config(), dim, T.HostParticles(dim, wl.pos, wl.vel, wl.types), precision=1) as s:
            n0 = s.lib.mps_launch_count()
            s.step(1)
            launches.append(s.lib.mps_launch_count() - n0)
            out.append(s.download())
            iters.append(s.metrics()["ppe_iterations"])
    assert iters[0] == iters[1]
    assert launches[1] - launches[0] == 1
    for f in ("pressure", "vel", "pos"):
        assert np.array_equal(out[0][f], out[1][f]), f


@pytest.mark.parametrize("solver,delta", [("0", "0.01"), ("1", "0.0001")])
def test_interval_of_the_reliable_updates(solver, delta, monkeypatch):
    _cuda()
    from mps_b200.session import start
    out, met = [], []
    for env in (None, delta):
        if env:
            monkeypatch.setenv("MPS_RELIABLE_DELTA", env)
        wl = _workload(3)
        wl.params["solver_type"] = solver
        with start(wl.config(), 3, T.HostParticles(3, wl.pos, wl.vel, wl.types), precision=1) as s:
            s.step(1)
            out.append(s.download())
            met.append(s.metrics())
    assert met[0]["converged"] == 1
    for k in ("ppe_outer", "ppe_iterations"):
        assert met[0][k] == met[1][k], k
    for f in ("pressure", "vel", "pos"):
        assert np.array_equal(out[0][f], out[1][f]), f
