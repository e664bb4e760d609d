"""The PPE's assembly by groups of lanes against the oracle, bit for bit.

Rows with every remainder of neighbours by the group's width, rows of
particles whose neighbours exceed the list's room (a second lattice inside the
fluid: walked by one lane), both dimensions, with and without the mixed form's
packed words and row sums; pressures within 1e-8.
"""
import ctypes as C

import numpy as np
import pytest

from test_gpu_lists import _workload
from test_gpu_parity import _cuda, _moved_state, _oracle, _rel, _session

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("doubled", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
def test_assembly_by_lanes(dim, doubled, precision):
    _cuda()
    wl = _workload(dim, doubled)
    orc = _oracle(dim)
    cfg, hp, nl, cl = _moved_state(wl, orc, steps=0, research=True)
    m = cfg.max_neighbors
    orc.lib.oracle_number_density(C.byref(hp.ps), C.byref(nl.nl), C.byref(cfg))
    orc.lib.oracle_judge_free_surface(C.byref(hp.ps), cfg.surface_threshold)   # known pressures: a regular system
    eq, rp, ci, va, b = orc.assemble(hp, nl, cfg)
    assert len(set(nl.count[: hp.n] % 8)) == 8
    ho = hp.copy()
    orc.lib.oracle_solve_pressure(C.byref(ho.ps), C.byref(nl.nl), C.byref(cfg))
    with _session(cfg, dim, hp, precision=precision) as s:
        s.set_initial_params(hp.ps.n0, hp.ps.lambda_, hp.ps.n0_count)
        s.run_stage("solve_pressure", nl.neighbors[: hp.n * m], nl.count[: hp.n], m)
        got = s.ppe()
        pressure = s.download()["pressure"]
    for a, o in zip(got, (eq, rp, ci, va, b)):
        assert np.array_equal(a, o)
    assert _rel(pressure, ho.view["pressure"]) < 1e-8
