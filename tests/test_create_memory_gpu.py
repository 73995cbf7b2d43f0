"""A context takes the FP64 mode's work space at creation only where that mode is on
and the lattice small enough for its first S(q,t) to be captured."""
from __future__ import annotations

import ctypes as C

import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu


def allocations(N, mode):
    """Device allocations of asd_ctx_create: the first injected failure it survives."""
    p = asd.Params.make(N, 4)
    lib = asd.load()
    try:
        for n in range(1, 100):
            asd.debug_fail_alloc(n)
            h = C.c_void_p()
            rc = lib.asd_ctx_create(C.byref(p), 1 << asd.MODES[mode], C.byref(h))
            if rc == asd.ASD_OK:
                lib.asd_ctx_destroy(h)
                return n - 1
            assert rc == asd.ASD_ERR_NOMEM
    finally:
        asd.debug_fail_alloc(0)
    raise AssertionError("never succeeded")


def test_fp64_work_space_only_where_it_is_used():
    small, large = 12, 45
    assert allocations(small, "fp64") == allocations(large, "fp64") + 2
    for mode in ("tf32x3", "bf16x3", "fp16x3"):
        assert allocations(small, mode) == allocations(large, mode)
