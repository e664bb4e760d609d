"""Device memory of the multilevel preconditioner.

Plain CG holds none of it: a session on a grid of many cells stays below 64
bytes a cell (the grid's own arrays take 11 ints and an eighth of room, 49.5
bytes, and the scans' workspace).  Where the device has no memory for the
nested grids' arrays, or for the operators on them, the step is the one of the
IC(0) form, bit for bit.
"""
import numpy as np
import pytest

from mps_b200 import _lib
from mps_b200 import types as T
from mps_b200 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "pressure", "n", "type", "on_surface")
MB = 1 << 20


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _free(torch):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _wide(dim, cells, **kw):
    """A small dam break in a domain of about `cells` cells."""
    wl = (W.small_dambreak3d if dim == 3 else W.small_dambreak2d)(l0=0.02, seed=13, **kw)
    side = cells ** (1.0 / dim) * 3.1 * 0.02
    for d in range(dim):
        wl.params["domain_%s_max" % "xyz"[d]] = repr(side)
    return wl


def _start(wl, **kw):
    from mps_b200.session import start
    return start(wl.config(), wl.dim, T.HostParticles(wl.dim, wl.pos, wl.vel, wl.types), **kw)


@pytest.mark.parametrize("dim", [2, 3])
def test_plain_cg_holds_no_nested_grids(dim):
    torch = _torch()
    cells = 2.0e7
    with _start(_wide(dim, 1000.0, solver_type=0)) as s:   # the context and the kernels
        s.step(1)
    wl = _wide(dim, cells, solver_type=0)
    before = _free(torch)
    with _start(wl) as s:
        s.step(1)
        used = before - _free(torch)
    assert 40.0 * cells < used < 64.0 * cells + 64 * MB


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("what", ["grids", "grids of a new session", "operators"])
def test_refused_memory_falls_back_to_ic0(what, precision, monkeypatch):
    torch = _torch()
    if what != "operators":
        wl, room = _wide(3, 4.0e7), 1024 * MB      # the grids' arrays take 40 bytes a node and more
    else:
        # wall particles beyond each other's reach, a cell each, around the dam: 4 kB a cell and 2 kB
        # a node for the operators, next to nothing for a factor
        wl, room = _wide(3, 60.0 ** 3), 200 * MB
        k = np.stack(np.meshgrid(*[np.arange(30)] * 3, indexing="ij"), -1).reshape(-1, 3)
        far = 1.0 + 0.08 * k
        wl.pos = np.concatenate([wl.pos, far])
        wl.vel = np.concatenate([wl.vel, np.zeros_like(far)])
        wl.types = np.concatenate([wl.types, np.full(len(far), T.WALL, np.int32)])
    monkeypatch.setenv("MPS_SWEEP", "0")
    with _start(wl, precision=precision) as s:
        s.step(1)
        want, met = s.download(), s.metrics()
    monkeypatch.delenv("MPS_SWEEP")
    with _start(wl, precision=precision) as s:
        s.step(1)   # multilevel
        got, m = s.download(), s.metrics()
        assert m["converged"] == 1 and m["ppe_iterations"] != met["ppe_iterations"]
    if what == "grids of a new session":   # its own grid takes 2.2 GB, these 2.4 more
        held = torch.empty(_free(torch) - 3500 * MB, dtype=torch.uint8, device="cuda")
        with _start(wl, precision=precision) as s:
            s.step(1)
            got, m = s.download(), s.metrics()
        del held
        torch.cuda.empty_cache()
        assert m["converged"] == 1 and m["ppe_iterations"] == met["ppe_iterations"]
        for f in FIELDS:
            assert np.array_equal(got[f], want[f]), f
        return
    wl.params["solver_type"] = "0"
    with _start(wl, precision=precision) as s:
        ck = torch.empty(s.state_bytes(), dtype=torch.uint8, device="cuda")
        s.state_save(ck.data_ptr())
        s.step(1)   # the arrays of the step itself
        s.state_load(ck.data_ptr())
        del ck
        s.params.solver_type = 1
        s._check(s.lib.mps_update_params(s.h, _lib.C.byref(s.params)))
        held = torch.empty(_free(torch) - room, dtype=torch.uint8, device="cuda")
        s.step(1)
        got, m = s.download(), s.metrics()
        del held
    torch.cuda.empty_cache()
    assert m["converged"] == 1 and m["ppe_iterations"] == met["ppe_iterations"]
    for f in FIELDS:
        assert np.array_equal(got[f], want[f]), f
