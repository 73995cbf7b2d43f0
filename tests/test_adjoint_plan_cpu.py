"""The CTAs per replica of the resident adjoint, without a GPU."""
from __future__ import annotations

import pytest

import asd_b200 as asd


@pytest.mark.parametrize("sms", [148, 132, 74, 1])
def test_plan_is_one_two_four_or_none(sms):
    plan = asd.load().asd_check_adjoint_ctas
    for N in range(3, 130):
        for nfile in (1, 15, 16, 17, 37, 74, 75, 148, 1000):
            ctas = plan(N, nfile, sms)
            assert (ctas in (1, 2, 4)) if 12 <= N <= 64 and nfile >= 16 else ctas == 0
            assert ctas != 1 or N <= 36  # a larger lattice does not fit one SM


def test_bad_arguments_give_none():
    plan = asd.load().asd_check_adjoint_ctas
    assert plan(0, 16, 148) == plan(32, 0, 148) == plan(32, 16, 0) == 0
