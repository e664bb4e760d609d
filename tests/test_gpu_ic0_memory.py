"""An IC(0) factor on request (the multilevel form's solve needs none) whose
arrays the device has no memory for, one after the other up to the FP32 copies:
an error each time, with nothing left half formed.  The call that succeeds
gives the factor and the application of a session that met no refusal.
"""
import numpy as np
import pytest

from mps_b200 import _lib
from mps_b200 import types as T
from mps_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_factor_after_refused_memory():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mps_b200.session import start
    wl = W.dambreak("c1", l0=0.0125, seed=8)
    room, r, want, refused = 96 << 20, None, None, 0
    for hog in (False, True):
        hp = T.HostParticles(3, wl.pos, wl.vel, wl.types)
        with start(wl.config(), 3, hp, precision=1) as s:
            s.step(1)
            rows = s.metrics()["n_eq"]
            r = np.random.default_rng(2).normal(size=rows)
            z = None
            while z is None:
                held = None
                if hog:
                    torch.cuda.empty_cache()
                    held = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
                try:
                    z = s.apply_preconditioner(r)
                except _lib.MpsError as e:
                    assert hog and e.code == -3
                    refused += 1
                    assert refused < 40
                del held
            f = s.ic0()
        torch.cuda.empty_cache()
        if not hog:
            want = (z, f)
    assert refused >= 3
    assert np.array_equal(z, want[0])
    for k in f:
        assert np.array_equal(f[k], want[1][k]), k
