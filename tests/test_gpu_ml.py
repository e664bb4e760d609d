"""The multilevel preconditioner of the PPE solve against the IC(0) form.

Both solve the same system, the IC(0) form (MPS_SWEEP=0) being pinned to the
oracle elsewhere; the pressures agree to the solver's rounding.  Cases: both
dimensions and precision forms, the additive and the multiplicative first
grid (MPS_ML_ADD), the V-cycle dense from the coarsest grid on and from the
first grid of at most 1,024 nodes on (MPS_ML_DENSE), grids of odd and even
extents, cells with up to ~90 unknowns, and the loop as launches and in one
cluster (MPS_ML_SMALL).  Tolerances: pressure 1e-8, velocity 1e-10 and
position 1e-14 relative L2 after one step, as for a step against the oracle.

A wall region that no known pressure bounds and no source reaches keeps the
zero pressure a zero start gives it, bit for bit, although coarse nodes couple
it to the fluid's.
"""
import numpy as np
import pytest

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


def _step(monkeypatch, wl, precision, steps=1, **env):
    from mps_b200.session import start
    for k in ("MPS_SWEEP", "MPS_ML_ADD", "MPS_ML_DENSE", "MPS_ML_SMALL"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    hp = T.HostParticles(wl.dim, wl.pos, wl.vel, wl.types)
    s = start(wl.config(), wl.dim, hp, precision=precision)
    try:
        s.step(steps)
        return s.download(), s.metrics()
    finally:
        s.close()


def _droplet():
    """A block of fluid hanging in a dry tank, further than the interaction
    radius from the walls but in cells next to theirs."""
    wl = W.small_dambreak3d(l0=0.02, seed=9, domain=(0.5, 0.5, 0.5), water=(0.3, 0.3, 0.3), jitter=0.0)
    keep = (wl.types != T.FLUID) | np.all(wl.pos > 0.0999, axis=1)
    wl.pos, wl.vel, wl.types = wl.pos[keep], wl.vel[keep], wl.types[keep]
    return wl


CASES = {
    "dam3d": lambda: W.dambreak("c1", l0=0.02, seed=3),
    "small3d": lambda: W.small_dambreak3d(l0=0.0171, seed=1),
    "dam2d": lambda: W.small_dambreak2d(l0=0.01, seed=4),
    "odd2d": lambda: W.small_dambreak2d(l0=0.0137, seed=6),
    "dense3d": lambda: W.small_dambreak3d(l0=0.014, seed=5, influence_ratio_lap="4.43"),
    "droplet": _droplet,
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_multilevel_matches_ic0(name, precision, monkeypatch):
    _cuda()
    wl = CASES[name]()
    ref, mref = _step(monkeypatch, wl, precision, MPS_SWEEP="0")
    for add in ("0", "1000000"):
        for dense in ("0", "150", "1024"):
            for small in ("0", "1000000"):
                g, m = _step(monkeypatch, wl, precision, MPS_ML_ADD=add, MPS_ML_DENSE=dense, MPS_ML_SMALL=small)
                assert m["converged"] == 1
                for f in ("n", "on_surface", "type"):
                    assert np.array_equal(g[f], ref[f]), f
                assert _rel(g["pressure"], ref["pressure"]) < 1e-8
                assert _rel(g["vel"], ref["vel"]) < 1e-10
                assert _rel(g["pos"], ref["pos"]) < 1e-14
                if name == "droplet":
                    wall = g["type"] == T.WALL
                    assert np.abs(g["pressure"]).max() > 0.0
                    assert np.all(g["pressure"][wall] == 0.0) and np.all(ref["pressure"][wall] == 0.0)


def test_multilevel_reruns_are_bit_identical(monkeypatch):
    _cuda()
    wl = W.dambreak("c1", l0=0.02, seed=6)
    for add in ("0", "1000000"):
        a, ma = _step(monkeypatch, wl, 0, steps=2, MPS_ML_ADD=add)
        b, mb = _step(monkeypatch, wl, 0, steps=2, MPS_ML_ADD=add)
        assert ma["ppe_iterations"] == mb["ppe_iterations"]
        for f in ("pressure", "pos", "vel"):
            assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("dim", [2, 3])
def test_ic0_survives_a_larger_grid(dim):
    """The IC(0) factor is formed on request; a domain enlarged in between
    (the grid's arrays are allocated anew) leaves it as it was."""
    _cuda()
    from mps_b200 import _lib
    from mps_b200.session import start
    wl = CASES["small3d" if dim == 3 else "dam2d"]()
    got = []
    for grow in (False, True):
        hp = T.HostParticles(dim, wl.pos, wl.vel, wl.types)
        s = start(wl.config(), dim, hp)
        try:
            s.step(1)
            if grow:
                for d in range(dim):
                    s.params.domain_max[d] *= 4.0
                s._check(s.lib.mps_update_params(s.h, _lib.C.byref(s.params)))
            got.append((s.ic0(), s.cell_blocks()))
        finally:
            s.close()
    (f0, c0), (f1, c1) = got
    for k in f0:
        assert np.array_equal(f0[k], f1[k]), k
    for a, b in zip(c0, c1):
        assert np.array_equal(a, b)
