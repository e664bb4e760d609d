"""mps_update_params on a session with a step behind it.

A refused change (a grid beyond 2^30 cells, or one the device has no memory
for) leaves the parameters and the grid of before: the next search and step
give the bits of a session that was never asked, the same change is refused
again, and a change that can be made is made.  A changed domain forms no IC(0)
factor; one asked for afterwards is the factor of the step before it.
"""
import numpy as np
import pytest

from mps_b200 import _lib
from mps_b200 import types as T
from mps_b200 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "pressure", "n", "type", "on_surface")


def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _session(dim, **kw):
    from mps_b200.session import start
    wl = (W.small_dambreak3d if dim == 3 else W.small_dambreak2d)(l0=0.02, seed=21)
    return start(wl.config(), dim, T.HostParticles(dim, wl.pos, wl.vel, wl.types), **kw)


def _update(s):
    s._check(s.lib.mps_update_params(s.h, _lib.C.byref(s.params)))


def _domain(s, dim, factor):
    for d in range(dim):
        s.params.domain_max[d] = factor[d] if isinstance(factor, list) else s.params.domain_max[d] * factor


@pytest.mark.parametrize("why", ["cells", "memory"])
@pytest.mark.parametrize("dim", [2, 3])
def test_refused_change_leaves_the_session_as_it_was(dim, why):
    torch = _cuda()
    with _session(dim) as s:
        s.step(1)
        s.neighbor_search()
        s.step(1)
        want = s.download()
    hog = None
    with _session(dim) as s:
        s.step(1)
        before = [s.params.domain_max[d] for d in range(dim)]
        re = 3.1 * 0.02
        # twice the cells there may be; or half of them, 20 GB and more of device memory
        cells = 2.0 ** 31 if why == "cells" else 2.0 ** 29
        if why == "memory":
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            free = torch.cuda.mem_get_info()[0]
            hog = torch.empty(free - (4 << 30), dtype=torch.uint8, device="cuda")
        side = cells ** (1.0 / dim) * re
        for _ in range(2):
            _domain(s, dim, [side] * dim)
            with pytest.raises(_lib.MpsError) as e:
                _update(s)
            assert e.value.code == (-1 if why == "cells" else -3)
        del hog
        torch.cuda.empty_cache()
        _domain(s, dim, before)
        s.neighbor_search()
        s.step(1)
        got = s.download()
        for f in FIELDS:
            assert np.array_equal(got[f], want[f]), f
        _domain(s, dim, 3.0)
        _update(s)
        s.neighbor_search()
        s.step(1)
        assert s.metrics()["converged"] == 1


@pytest.mark.parametrize("precision", [0, 1])
def test_changed_domain_forms_no_factor(precision):
    _cuda()
    got = []
    for grow in (0, 1, 2):
        with _session(3, precision=precision) as s:
            s.step(1)
            n0 = s.lib.mps_launch_count()
            for _ in range(grow):
                _domain(s, 3, 2.0)
                _update(s)
            assert s.lib.mps_launch_count() == n0
            f = s.ic0()
            r = np.random.default_rng(3).normal(size=len(f["b"]))
            got.append((f, s.cell_blocks(), s.apply_preconditioner(r)))
    for f, blocks, z in got[1:]:
        for k in f:
            assert np.array_equal(f[k], got[0][0][k]), k
        for a, b in zip(blocks, got[0][1]):
            assert np.array_equal(a, b)
        assert np.array_equal(z, got[0][2])
