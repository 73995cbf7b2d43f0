"""The drop-in functions' copies of pageable arrays: plain below 2 MB, staged by
several threads in 1 MB chunks above.  Replicas are independent, so a staged call
must equal, bit for bit, the same replicas in calls small enough for plain copies;
sizes just below and above the limit, whole chunks and remainders."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu

REPLICA = 32 * 32 * 3 * 8  # bytes of a 32 x 32 replica: 24 KB


@pytest.mark.parametrize("nfile", [17, 18, 85, 86, 128, 171, 300])
def test_staged_equals_plain(nfile):
    """euler uploads and downloads nfile * 24 KB (staged from 86 replicas),
    runge_kutta downloads five times that in one go (staged from 18)."""
    N = 32
    s = asd.random_spins(N, nfile, seed=nfile)
    asd.set_params(N, nfile, 1.0, 0.02)
    d = asd.euler(s)
    rk = asd.runge_kutta(s)
    asd.set_params(N, 1, 1.0, 0.02)
    for f in sorted({0, 1, nfile // 2, nfile - 2, nfile - 1}):
        one = s[f:f + 1]
        assert np.array_equal(d[f:f + 1], asd.euler(one)), f
        for got, want in zip(rk, asd.runge_kutta(one)):
            assert np.array_equal(got[f:f + 1], want), f
    assert not np.isnan(d).any() and not any(np.isnan(r).any() for r in rk)
