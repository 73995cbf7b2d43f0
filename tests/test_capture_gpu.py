"""Calls captured into a CUDA graph and replayed: the steps go on from where the
last replay left the spins, and S(q,t) is that of the state and the origin at the
time of the replay, bit for bit what the same calls give one by one.  Sizes: S(q,t)
in FP64 captured as the first call on a small lattice, resident steps of one SM and
of a cluster, stage kernels, and lattices whose uncaptured steps alternate between
two buffers."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KW = dict(J1=-1.0, alpha=0.1, dt=0.01)


def eager(N, nfile, s0, origin, replays, nsteps):
    """S(q,t) and the spins after each of `replays` runs of nsteps steps from s0."""
    out = []
    with asd.Context(asd.Params.make(N, nfile, **KW), modes=["fp64"]) as ctx:
        ctx.set_spins(origin, as_origin=True)
        ctx.set_spins(s0, as_origin=False)
        for _ in range(replays):
            ctx.step(nsteps)
            out.append((ctx.sqt("fp64"), np.array(ctx.get_spins()).reshape(-1)))
    return out


@pytest.mark.parametrize("N,nfile,nsteps", [(12, 16, 1), (32, 40, 3), (64, 20, 2), (100, 24, 4),
                                            (160, 4, 1), (160, 16, 1), (128, 30, 1), (256, 8, 1)])
def test_replayed_steps_and_sqt(N, nfile, nsteps):
    a, b = (asd.random_spins(N, nfile, seed=N + k) for k in (0, 1))
    stream = torch.cuda.Stream()
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    spins = torch.zeros(nfile * N * N * 3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with asd.Context(asd.Params.make(N, nfile, **KW), modes=["fp64"]) as ctx:
        ctx.set_stream(stream.cuda_stream)
        ctx.set_spins(a, as_origin=True)
        if N > 39:  # the first S(q,t) of a larger lattice takes work space
            ctx.sqt("fp64")
        ctx.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.step(nsteps)
            ctx.sqt_async("fp64", out.data_ptr())
            ctx.get_spins_device(spins.data_ptr())
        for origin, start in ((a, a), (b, a)):  # the second time with another origin
            ctx.set_spins(origin, as_origin=True)
            ctx.set_spins(start, as_origin=False)
            ctx.synchronize()
            for s, y in eager(N, nfile, start, origin, 3, nsteps):
                with torch.cuda.stream(stream):
                    graph.replay()
                stream.synchronize()
                assert complex(*out.tolist()) == s
                assert np.array_equal(spins.cpu().numpy(), y)
        # and the uncaptured call still sees its own origin
        ctx.set_spins(a, as_origin=True)
        with asd.Context(asd.Params.make(N, nfile, **KW), modes=["fp64"]) as other:
            other.set_spins(a, as_origin=True)
            assert ctx.sqt("fp64") == other.sqt("fp64")
        del graph
