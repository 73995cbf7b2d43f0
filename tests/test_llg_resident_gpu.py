"""The resident RK4 steps (a replica's lattice on one SM or a cluster of SMs for
any number of steps; the default where they are the fastest) against the
oracle, bit for bit (tolerance 0), at the sizes where the kernel's geometry
changes: lattice sides at and around 32, 64 and 128 columns, sides that leave
threads idle or rows ragged, clusters with uneven rows, every combination of the
model's terms, |J1| = 1 (exchange added before J1 is applied) and not, one and
several steps a launch, and more replicas than fit the GPU at once."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd
import oracle as orc

pytestmark = pytest.mark.gpu

MODELS = [dict(J1=1.0, dt=0.02), dict(J1=-1.0, alpha=0.05, h=(0.1, -0.2, 0.5), dt=0.005),
          dict(J1=0.8, J2=0.2, alpha=0.1, dt=0.01), dict(J1=-1.0, J2=-0.3, dt=0.01),
          dict(J1=1.3, h=(0.0, 0.0, 0.4), dt=0.01)]


def lib_resident(N, nfile, nsteps, kw):
    """The default choice stays resident for these sizes: one launch for all steps."""
    s0 = asd.random_spins(N, nfile, seed=N + nfile)
    with asd.Context(asd.Params.make(N, nfile, **kw), modes=["fp64"]) as ctx:
        ctx.set_spins(s0, as_origin=True)
        ctx.step(nsteps)
        launches = ctx.last_launches()
        st = ctx.get_spins()
    return s0, st, launches


@pytest.mark.parametrize("model", range(len(MODELS)))
@pytest.mark.parametrize("N", [3, 5, 12, 31, 32, 33, 47, 63, 64])
def test_one_cta_per_replica(oracle, N, model):
    nfile, nsteps = 30 if N <= 33 else 100, 12
    s0, st, launches = lib_resident(N, nfile, nsteps, MODELS[model])
    assert launches == 1  # otherwise this would not test the resident kernel
    want = oracle.steps(orc.make_params(N, nfile, **MODELS[model]), s0, nsteps)
    assert np.array_equal(st, want)


@pytest.mark.parametrize("N,nfile,model", [(65, 70, 0), (96, 120, 1), (101, 70, 3), (128, 70, 1),
                                           (128, 70, 2)])
def test_clusters_per_replica(oracle, N, nfile, model):
    nsteps = 12
    s0, st, launches = lib_resident(N, nfile, nsteps, MODELS[model])
    assert launches == 1
    want = oracle.steps(orc.make_params(N, nfile, **MODELS[model]), s0, nsteps)
    assert np.array_equal(st, want)


@pytest.mark.parametrize("N,nfile,nsteps", [(8, 1000, 3), (32, 500, 1), (64, 160, 6), (64, 100, 1)])
def test_more_replicas_than_resident_and_single_steps(oracle, N, nfile, nsteps):
    kw = MODELS[1]
    s0, st, launches = lib_resident(N, nfile, nsteps, kw)
    assert launches == 1
    want = oracle.steps(orc.make_params(N, nfile, **kw), s0, nsteps)
    assert np.array_equal(st, want)


def test_zero_signs_survive():
    """A ferromagnet along z under J1 = -1: the exchange field's x and y sums are
    zeros, whose sign the |J1| = 1 form must keep as the stage kernels have it."""
    N, nfile = 16, 6
    up = np.zeros((nfile, N * N, 3))
    up[..., 2] = 1.0
    up[:, ::3, 0] = -0.0
    for J1 in (1.0, -1.0):
        out = {}
        for kern in ("auto", "stages"):
            with asd.Context(asd.Params.make(N, nfile, J1=J1, alpha=0.1, dt=0.01),
                             modes=["fp64"]) as ctx:
                ctx.set_llg_kernel(kern)
                ctx.set_spins(up, as_origin=True)
                ctx.step(5)
                out[kern] = ctx.get_spins()
        assert out["auto"].tobytes() == out["stages"].tobytes()
