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


PRELOAD = r"""
#include <cstdlib>
#include <new>
static thread_local int armed = 0;
extern "C" void fail_new(int on) { armed = on; }
void *operator new(std::size_t n) {
    void *p = armed ? nullptr : std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
"""

CHILD = r"""
import ctypes as C, sys
import numpy as np
import asd_b200 as asd
N, NFILE = 32, 120
spin = asd.random_spins(N, NFILE, seed=5).reshape(-1)
asd.set_params(N, NFILE, 1.0, 0.02)
runs = []
for failing in (0, 1):
    outs = [np.zeros_like(spin) for _ in range(5)]
    p = [C.c_void_p(x.ctypes.data) for x in (spin, *outs)]
    C.CDLL(None).fail_new(failing)
    asd.load().runge_kutta(*p)
    C.CDLL(None).fail_new(0)
    runs.append(outs)
assert all(np.array_equal(x, y) and x.any() for x, y in zip(*runs))
print("same")
"""


def test_no_exception_leaves_the_c_entry(tmp_path):
    """With every C++ allocation of the calling thread failing, runge_kutta still
    gives its results: the staging starts no threads and throws nothing."""
    import os
    import subprocess
    import sys

    src, lib = tmp_path / "fail_new.cpp", tmp_path / "fail_new.so"
    src.write_text(PRELOAD)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    env = dict(os.environ, LD_PRELOAD=str(lib),
               PYTHONPATH=os.pathsep.join([p for p in sys.path if p]))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
