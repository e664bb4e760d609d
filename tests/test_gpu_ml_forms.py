"""Which form of the multilevel solve runs, and that each of them does.

With profiling on, the metrics tell the loop in one cluster (one launch per
solve or stretch) from the loop of launches.  Its kernels differ by the lanes a
cell gets (16 for short rows, 32 for small cells, 64), by whether the matrix
fits the cluster's shared memory and by whether the cells take more than one
round: the cases reach all of these, in both matrix forms, and agree with the
loop of launches (pressure 1e-8, velocity 1e-10, position 1e-14).  A first
grid that is neither dense nor additive, or vectors beyond the shared memory,
leave the launches.
"""
import numpy as np
import pytest

from mps_b200 import types as T
from mps_b200 import workloads as W

pytestmark = pytest.mark.gpu

CTAS, WARPS, SMEM = 16, 32, 216 * 1024

CASES = {
    "2d": lambda: W.small_dambreak2d(l0=0.01, seed=4),
    "2d-many-cells": lambda: W.small_dambreak2d(l0=0.005, seed=4),
    "3d": lambda: W.small_dambreak3d(l0=0.02, seed=2),
    "3d-larger": lambda: W.dambreak("c1", l0=0.035, seed=2),
    "3d-wide-radius": lambda: W.small_dambreak3d(l0=0.014, seed=5, influence_ratio_lap="4.43"),
    "3d-wide-radius-small": lambda: W.small_dambreak3d(l0=0.03, seed=5, influence_ratio_lap="4.43"),
    "3d-small-cells": lambda: W.small_dambreak3d(l0=0.016, seed=5, influence_ratio_lap="2.6"),
}


def _step(monkeypatch, wl, precision, **env):
    from mps_b200.session import start
    for k in ("MPS_ML_ADD", "MPS_ML_DENSE", "MPS_ML_SMALL"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    with start(wl.config(), wl.dim, T.HostParticles(wl.dim, wl.pos, wl.vel, wl.types), precision=precision) as s:
        s.set_profiling()
        s.step(1)
        out, m = s.download(), s.metrics()
        m["cells"] = len(s.cell_blocks()[0])
    assert m["converged"] == 1
    return out, m


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("precision", [0, 1])
def test_every_kernel_of_the_cluster_loop_runs(precision, monkeypatch):
    _cuda()
    lanes, fits, rounds = set(), set(), set()
    for name, make in CASES.items():
        wl = make()
        ref, mref = _step(monkeypatch, wl, precision, MPS_ML_SMALL="0")
        got, m = _step(monkeypatch, wl, precision)
        assert mref["prof_pcg_launches"] == 0 and mref["prof_spmv_launches"] > 0, name
        assert m["prof_pcg_launches"] > 0 and m["prof_spmv_launches"] == 0, (name, m["n_eq"])
        for f, tol in (("pressure", 1e-8), ("vel", 1e-10), ("pos", 1e-14)):
            assert np.linalg.norm(got[f] - ref[f]) <= tol * np.linalg.norm(ref[f]), (name, f)
        w = 16 if m["nnz"] < 48 * m["n_eq"] else 32 if m["n_eq"] < 24 * m["cells"] else 64
        lanes.add(w)
        rounds.add(m["cells"] > CTAS * WARPS * 32 // w)
        entry = 8 if precision else 12
        if m["nnz"] / CTAS * 1.25 + 64 < (SMEM - 16 * m["n_eq"]) / entry:
            fits.add("yes")
        elif m["nnz"] / CTAS > (SMEM - 8 * m["n_eq"]) / entry:
            fits.add("no")
    assert lanes == {16, 32, 64} and rounds == {False, True} and fits == {"yes", "no"}


def _grid_nodes(wl):
    """Nodes in use on the first and the second grid: the corners of the cells
    that hold unknowns, and their parents."""
    from mps_b200 import config as CF
    from mps_b200.session import start
    cfg = wl.config()
    with start(cfg, wl.dim, T.HostParticles(wl.dim, wl.pos, wl.vel, wl.types)) as s:
        s.step(1)
        cell, p = s.cell_index(), s.download()
    re = CF.neighbor_radius(cfg)
    dims = [int(((cfg.domain_max[d] + 4.0 * re) - (cfg.domain_min[d] - 4.0 * re)) / re) + 2 for d in range(wl.dim)]
    unknown = ((p["type"] == T.FLUID) & (p["on_surface"] == 0)) | (p["type"] == T.WALL)
    c = np.unique(cell[unknown])
    xyz = np.stack(np.unravel_index(c, dims[::-1])[::-1], -1)
    bits = np.stack(np.meshgrid(*[[0, 1]] * wl.dim, indexing="ij"), -1).reshape(-1, wl.dim)
    first = np.unique((xyz[:, None, :] + bits[None]).reshape(-1, wl.dim), axis=0)
    second = np.unique(((first[:, None, :] + bits[None]) // 2).reshape(-1, wl.dim), axis=0)
    return len(first), len(second)


@pytest.mark.parametrize("form", ["steps", "dense", "additive", "too many unknowns"])
def test_rule_of_the_cluster_loop(form, monkeypatch):
    _cuda()
    wl = CASES["3d"]()
    na, nb = _grid_nodes(wl)
    assert 64 < nb < na <= 1024
    env = {"steps": dict(MPS_ML_DENSE=str(nb), MPS_ML_ADD="0"),             # a first grid by steps
           "dense": dict(MPS_ML_DENSE=str(na), MPS_ML_ADD="0"),             # dense from the first grid on
           "additive": dict(MPS_ML_DENSE=str(nb), MPS_ML_ADD="1000000"),    # dense from the second on
           "too many unknowns": dict(MPS_ML_SMALL="100")}[form]
    _, m = _step(monkeypatch, wl, 0, **env)
    assert (m["prof_pcg_launches"] > 0) == (form in ("dense", "additive"))


def test_vectors_beyond_the_shared_memory_leave_the_launches(monkeypatch):
    _cuda()
    _, m = _step(monkeypatch, W.dambreak("c1", l0=0.02, seed=3), 0, MPS_ML_SMALL="1000000", MPS_ML_ADD="1000000")
    assert 8 * m["n_eq"] < SMEM < 8 * m["n_eq"] + 16 * 1024 and m["prof_pcg_launches"] == 0
