"""Large transfers with pageable host memory (chunks moved by host threads).

Particle arrays around the size where the chunked path begins and around whole
numbers of its 1 MiB chunks come back byte for byte; a neighbour list large
enough for it drives the same step as the same list in page-locked memory, is
returned the same into either, and an index outside the particles in it is
reported.
"""
import ctypes as C

import numpy as np
import pytest

from mps_b200 import types as T
from mps_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("dim,num", [(3, 1), (3, 40329), (3, 40330), (3, 50412), (3, 90001), (2, 52428), (2, 52429),
                                     (2, 200003)])
def test_particles_round_trip(dim, num):
    _cuda()
    from mps_b200.session import Session
    wl = W.small_dambreak3d() if dim == 3 else W.small_dambreak2d()
    rng = np.random.default_rng(num)
    hp = T.HostParticles(dim, rng.random((num, dim)), rng.random((num, dim)), np.zeros(num, np.int32))
    for f in ("acc", "pressure", "n"):
        hp.arr[f] = rng.random(hp.arr[f].shape)
    want = hp.arr.copy()
    with Session(wl.config(), dim, num) as s:
        s.upload(hp)
        assert np.array_equal(s.download(), want)
        assert np.array_equal(s.pressure(), want["pressure"])
        s.upload_soa(want["pos"], want["vel"], want["type"])
        got = s.download()
        assert np.array_equal(got["pos"], want["pos"]) and np.array_equal(got["vel"], want["vel"])


def test_large_pageable_list_matches_page_locked():
    _cuda()
    import torch
    from mps_b200 import _lib
    from mps_b200.session import Session
    wl = W.dambreak("c1", l0=0.018, seed=12)
    cfg = wl.config()
    hp = T.HostParticles(3, wl.pos, wl.vel, wl.types)
    m, n = cfg.max_neighbors, hp.n
    with Session(cfg, 3, n) as s:
        s.upload(hp)
        n0 = s.compute_initial_params()
        s.neighbor_search()
        nb, cnt = s.neighbor_list(m)
        assert 4 * int(cnt.sum()) > (4 << 20)
        locked = torch.zeros(n * m, dtype=torch.int32, pin_memory=True)
        cl = torch.zeros(n, dtype=torch.int32, pin_memory=True)
        s._check(s.lib.mps_get_neighbor_list(s.h, locked.data_ptr(), cl.data_ptr(), m))
        a, b = nb.reshape(n, m), locked.numpy().reshape(n, m)
        assert np.array_equal(cnt, cl.numpy())
        used = np.arange(m)[None, :] < cnt[:, None]
        assert np.array_equal(a[used], b[used])
        out = []
        for lst in (nb, locked.numpy()):
            s.upload(hp)
            s.set_initial_params(*n0)
            s.step_with_list(lst, cnt, m)
            out.append(s.download())
        for f in ("pos", "vel", "pressure", "n", "type", "on_surface"):
            assert np.array_equal(out[0][f], out[1][f]), f
        bad = nb.copy()
        bad[(n - 1) * m] = n
        s.upload(hp)
        with pytest.raises(_lib.MpsError) as e:
            s.step_with_list(bad, cnt, m)
        assert e.value.code == -5 and cnt[n - 1] > 0
        assert C.sizeof(C.c_int) == 4
