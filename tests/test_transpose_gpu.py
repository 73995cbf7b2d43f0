"""The layout transposes behind set and get: every site, replica and component
comes back where it was, bit for bit, with full and ragged blocks of 32 sites and
32 replicas, and the site-major state in between is the one that S(q,t) and a
step in chunks of replicas read."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nfile", [(3, 1), (4, 31), (5, 32), (7, 33), (8, 64), (12, 100), (45, 33),
                                     (64, 7)])
def test_spins_come_back(N, nfile):
    s = np.arange(nfile * N * N * 3, dtype=np.float64).reshape(nfile, N * N, 3) + 0.25
    with asd.Context(asd.Params.make(N, nfile)) as ctx:
        ctx.set_spins(s, as_origin=True)
        assert np.array_equal(np.asarray(ctx.get_spins()).reshape(s.shape), s)


@pytest.mark.parametrize("N,nfile", [(12, 65), (20, 100), (13, 97)])
def test_steps_in_chunks_of_replicas(N, nfile):
    s = asd.random_spins(N, nfile, seed=N)
    kw = dict(J1=-1.0, alpha=0.1, dt=0.01)
    with asd.Context(asd.Params.make(N, nfile, **kw)) as ctx:
        ctx.set_spins(s, as_origin=True)
        ctx.step(1)
        want = np.array(ctx.get_spins())
    with asd.Context(asd.Params.make(N, nfile, **kw)) as ctx:
        ctx.set_spins(s, as_origin=True)
        buf = np.ascontiguousarray(s)
        got = np.zeros_like(buf)
        ctx.step_host(buf.ctypes.data, got.ctypes.data, "fp16x3")
    assert np.array_equal(got.reshape(want.shape), want)
