"""The drop-in entry points on host arrays other than separate pageable ones, at
sizes where copies go through the pinned chunks: the results of plain copies."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N, NFILE = 32, 120  # 2.9 MB an array


def rk(spin, outs):
    asd.set_params(N, NFILE, 1.0, 0.02)
    p = [C.c_void_p(x if isinstance(x, int) else x.ctypes.data) for x in (spin, *outs)]
    asd.load().runge_kutta(*p)


@pytest.fixture(scope="module")
def separate():
    spin = asd.random_spins(N, NFILE, seed=5).reshape(-1)
    outs = [np.zeros_like(spin) for _ in range(5)]  # cur, k1 .. k4
    rk(spin, outs)
    return spin, outs


def test_outputs_that_overlap_are_written_in_order(separate):
    spin, outs = separate
    n = spin.size
    for starts in ((0, n, n, n, 3 * n), (0, n // 2, n, 3 * n // 2, 2 * n), (0, 0, 0, 0, 0)):
        buf = np.zeros(4 * n)
        want = np.zeros(4 * n)
        for s, o in zip(starts, outs):
            want[s:s + n] = o
        rk(spin, [buf[s:s + n] for s in starts])
        assert np.array_equal(buf, want), starts


def test_page_locked_and_managed_arrays(separate):
    from cuda.bindings import runtime as rt

    spin, outs = separate
    locked = [torch.zeros(spin.size, dtype=torch.float64).pin_memory().numpy() for _ in range(6)]
    locked[0][:] = spin
    rk(locked[0], locked[1:])
    for got, want in zip(locked[1:], outs):
        assert np.array_equal(got, want)
    ptrs = []
    try:
        for _ in range(6):
            err, p = rt.cudaMallocManaged(spin.nbytes, rt.cudaMemAttachGlobal)
            assert int(err) == 0
            ptrs.append(int(p))
        managed = [np.frombuffer((C.c_char * spin.nbytes).from_address(p)) for p in ptrs]
        managed[0][:] = spin
        rk(ptrs[0], ptrs[1:])
        for got, want in zip(managed[1:], outs):
            assert np.array_equal(got, want)
    finally:
        for p in ptrs:
            rt.cudaFree(p)


def test_null_arrays_are_refused_as_before(separate):
    """A null input or output: reported, nothing read or written through it."""
    spin, outs = separate
    new = [np.zeros_like(spin) for _ in range(5)]
    rk(0, new)
    assert "invalid" in asd.last_error()
    assert all((x == 0.0).all() for x in new)
    rk(spin, [new[0], 0, *new[2:]])
    assert "invalid" in asd.last_error()
    rk(spin, new)
    for got, want in zip(new, outs):
        assert np.array_equal(got, want)
