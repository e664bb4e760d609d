"""Profiling on or off, a step launches the same kernels and gives the same
bits, in every loop of the solver: small systems (the loop in one cluster),
larger ones (launches), plain CG, and the IC(0) forms.  Every iteration is in
the profiling metrics once.
"""
import numpy as np
import pytest

from mps_b200 import types as T
from mps_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("loop", ["cluster", "launches", "cg", "ic0", "persistent"])
def test_profiling_changes_nothing(loop, precision, monkeypatch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mps_b200.session import start
    wl = W.small_dambreak3d(l0=0.02, seed=19, solver_type=0 if loop == "cg" else 1)
    if loop in ("ic0", "persistent"):
        monkeypatch.setenv("MPS_SWEEP", "0" if loop == "ic0" else "2")
    if loop == "launches":
        monkeypatch.setenv("MPS_ML_SMALL", "0")
    out, met, launches = [], [], []
    for on in (False, True):
        with start(wl.config(), 3, T.HostParticles(3, wl.pos, wl.vel, wl.types), precision=precision) as s:
            s.set_profiling(on)
            n0 = s.lib.mps_launch_count()
            s.step(2)
            launches.append(s.lib.mps_launch_count() - n0)
            out.append(s.download())
            met.append(s.metrics())
    for f in ("pos", "vel", "pressure", "n", "type", "on_surface"):
        assert np.array_equal(out[0][f], out[1][f]), f
    assert launches[0] == launches[1]
    assert met[0]["total_iterations"] == met[1]["total_iterations"] > 0
    assert met[0]["prof_iterations"] == 0
    m = met[1]
    assert m["prof_iterations"] == m["total_iterations"]
    whole = loop in ("cluster", "persistent")
    assert (m["prof_pcg_iterations"], m["prof_pcg_launches"] > 0) == (m["total_iterations"] if whole else 0, whole)
    assert (m["prof_pcg_ms"] > 0.0) == whole and (m["prof_vec_ms"] > 0.0) != whole


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("form", ["add", "mult", "dense"])
def test_serial_launches_give_the_same_bits(form, precision, monkeypatch):
    """The multilevel loop's launches one after the other (MPS_PDL_MASK=0) and
    as programmatic dependents: whole (6), and either group alone."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mps_b200.session import start
    wl = W.dambreak("c1", l0=0.02, seed=4)
    monkeypatch.setenv("MPS_ML_SMALL", "0")
    monkeypatch.setenv("MPS_ML_ADD", "1000000" if form == "add" else "0")
    monkeypatch.setenv("MPS_ML_DENSE", "1024" if form == "dense" else "64")
    out = []
    for mask in ("6", "0", "2", "4"):
        monkeypatch.setenv("MPS_PDL_MASK", mask)
        with start(wl.config(), 3, T.HostParticles(3, wl.pos, wl.vel, wl.types), precision=precision) as s:
            s.step(2)
            out.append((s.download(), s.metrics()["total_iterations"]))
    for g, it in out[1:]:
        assert it == out[0][1]
        for f in ("pos", "vel", "pressure"):
            assert np.array_equal(g[f], out[0][0][f]), f
