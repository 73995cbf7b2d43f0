"""The work that users of asd-b200 have it do, as cases that can be timed.

    listed()             the cases, dicts of plain values
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call: spins on the GPU
                         (or in host memory), a context, output buffers
    run(state)           one pass through the public entry points
    work(case)           bytes and operations that the pass cannot do without
    exact(case, seed)    the same outputs from plain torch in 64 bits

Kinds of work:

    series  a simulation that evaluates S(q,t) at one q every `stride` steps,
            in one of the four modes, and takes its spins at the end
            (asd_ctx_step, asd_ctx_sqt_async, asd_ctx_get_spins_device)
    grid    the same with S(q,t) on the whole q grid (asd_ctx_sqt_grid_async)
    llg     time stepping alone, the new spins handed to the caller's device
            buffer (asd_ctx_step, asd_ctx_get_spins_device)
    loss    parameter fitting: loss and gradient by the adjoint
            (asd_ctx_loss_grad)
    batch   lattices of several sizes in one launch (asd_batch_run), their
            spins read back
    host    steps on pinned host buffers (asd_ctx_step_host_async)
    dropin  one step of the reference's program through its own entry points
            on pageable host arrays (runge_kutta, fused_dgemm)
"""
from __future__ import annotations

import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "asd-kernel-fusion_b200"))

import asd_b200 as asd  # noqa: E402

MODES = ("fp64", "tf32x3", "bf16x3", "fp16x3")
BATCH_SIDES = (48, 64, 96, 128, 160)


def _case(kind, **kw):
    base = dict(kind=kind, N=0, nfile=0, J1=1.0, J2=0.0, alpha=0.0, hz=0.0, dt=0.005)
    base.update(kw)
    return base


def listed():
    af = dict(J1=-1.0, alpha=0.05, hz=0.5, dt=0.005)      # the 128 x 128 antiferromagnet
    j2 = dict(J1=1.0, J2=-0.3, alpha=0.02, dt=0.005)      # the 256 x 256 lattice with J2
    cases = {
        # the smallest runs: launches and latency count.  The plain method on a
        # 32 x 32 lattice with 200 snapshots, the whole q grid after every step
        "plain_grid_32": _case("grid", N=32, nfile=200, J1=1.0, alpha=0.1, dt=0.01, mode="fp64",
                               stride=1, evals=8),
        # the reference's own model (no damping, no field) on an odd lattice
        # side and a ragged replica count, S(q,t) in FP64 every 5 steps
        "series_fp64_51": _case("series", N=51, nfile=70, J1=1.0, dt=0.02, mode="fp64", stride=5,
                                evals=4),
        # a small ensemble stepped far between two looks at its spins
        "llg_64": _case("llg", N=64, nfile=100, J1=1.0, alpha=0.1, hz=0.2, dt=0.01, nsteps=50),
        # ordinary sizes: the antiferromagnet with 500 snapshots, plain against
        # split precision, and its time stepping alone
        "series_fp64_128": _case("series", N=128, nfile=500, mode="fp64", stride=1, evals=1, **af),
        "series_tf32x3_128": _case("series", N=128, nfile=500, mode="tf32x3", stride=1, evals=4,
                                   **af),
        "llg_128": _case("llg", N=128, nfile=500, nsteps=10, **af),
        # the whole q grid in split precision on a lattice of ragged tiles
        "grid_fp16x3_100": _case("grid", N=100, nfile=240, mode="fp16x3", stride=1, evals=2, **af),
        # the largest: 256 x 256 with 1000 snapshots and J2, one step with S(q,t)
        "series_bf16x3_256": _case("series", N=256, nfile=1000, mode="bf16x3", stride=1, evals=1,
                                   **j2),
        # fitting J, alpha and h to a target S(q,t): forward and adjoint
        "loss_64": _case("loss", N=64, nfile=100, J1=0.8, alpha=0.15, hz=0.0, dt=0.01, nsteps=100,
                         stride=10, checkpoint=50),
        # an ensemble of 48 lattices of uneven size, damping and noise
        "batch_48": _case("batch", count=48, nsteps=500, sizes_seed=0, dt=0.01),
        # a program that keeps its spins in host memory, steps pipelined
        "host_128": _case("host", N=128, nfile=500, mode="tf32x3", nsteps=4, **af),
        # the reference's fused program: 80 snapshots is its largest valid K
        "dropin_32": _case("dropin", N=32, nfile=80, J1=1.0, dt=0.02),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _model(rng):
    """Parameters of one of the models in use, each term switched on or off."""
    return dict(J1=rng.choice((1.0, -1.0, 0.8)), J2=rng.choice((0.0, 0.0, -0.3, 0.2)),
                alpha=rng.choice((0.0, 0.02, 0.05, 0.1)), hz=rng.choice((0.0, 0.2, 0.5)),
                dt=rng.choice((0.005, 0.01)))


def draw(rng):
    kind = rng.choice(("series", "series", "grid", "llg", "llg", "loss", "batch", "host", "dropin"))
    if kind in ("series", "grid"):
        N, nf = _logint(rng, 12, 160), _logint(rng, 8, 500)
        evals, stride = rng.randint(1, 8), rng.randint(1, 6)
        while 6.0 * N ** 4 * nf * evals > 6e11:  # products of the correlation GEMM
            nf, evals = max(8, int(nf * 0.7)), max(1, evals - 1)
            if nf == 8 and evals == 1:
                N = int(N * 0.9)
        return _case(kind, N=N, nfile=nf, mode=rng.choice(MODES), stride=stride, evals=evals,
                     **_model(rng))
    if kind == "llg":
        N, nf = _logint(rng, 12, 256), _logint(rng, 4, 1000)
        nsteps = _logint(rng, 1, 50)
        while float(N) * N * nf * nsteps > 1.3e8:
            nf, nsteps = max(4, int(nf * 0.7)), max(1, int(nsteps * 0.8))
        return _case(kind, N=N, nfile=nf, nsteps=nsteps, **_model(rng))
    if kind == "loss":
        stride = rng.randint(2, 12)
        return _case(kind, N=_logint(rng, 12, 64), nfile=_logint(rng, 8, 100),
                     nsteps=stride * rng.randint(2, 100 // stride), stride=stride,
                     checkpoint=rng.choice((10, 25, 50)), **_model(rng))
    if kind == "batch":
        return _case(kind, count=rng.randint(8, 48), nsteps=_logint(rng, 50, 500),
                     sizes_seed=rng.randrange(1 << 20), dt=rng.choice((0.005, 0.01)))
    if kind == "host":
        N, nf = _logint(rng, 16, 128), _logint(rng, 8, 500)
        return _case(kind, N=N, nfile=nf, mode=rng.choice(MODES[1:] if N > 64 else MODES),
                     nsteps=rng.randint(2, 4), **_model(rng))
    return _case("dropin", N=2 * rng.randint(6, 18), nfile=_logint(rng, 4, 80), J1=1.0, dt=0.02)


# ------------------------------------------------------------------- inputs
def _spins(case, seed, salt=0):
    """Spins uniform on the sphere, [nfile][N*N][3] float64 on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)
    shape = (case["nfile"], case["N"] * case["N"])
    z = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64).mul_(2.0).sub_(1.0)
    phi = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64).mul_(2.0 * math.pi)
    s = torch.empty(shape + (3,), device="cuda", dtype=torch.float64)
    r = (1.0 - z * z).sqrt_()
    s[..., 0] = r * phi.cos()
    s[..., 1] = r * phi.sin_()
    s[..., 2] = z
    return s


def _params(case, **over):
    c = dict(case, **over)
    return asd.Params.make(c["N"], c["nfile"], J1=c["J1"], J2=c["J2"], alpha=c["alpha"],
                           h=(0.0, 0.0, c["hz"]), dt=c["dt"])


def _lattices(case):
    """(N, noise amplitude, alpha) of the batch's lattices."""
    rng = random.Random(case["sizes_seed"])
    return [(rng.choice(BATCH_SIDES), rng.uniform(0.0, 0.5), rng.uniform(0.01, 0.2))
            for _ in range(case["count"])]


def _batch_spins(case, seed):
    """Per lattice float32 [N*N][3]: ordered along z with Gaussian noise, normalised."""
    rng = np.random.default_rng(seed)
    out = []
    for n, eta, _ in _lattices(case):
        s = eta * rng.standard_normal((n * n, 3))
        s[:, 2] += 1.0
        s /= np.linalg.norm(s, axis=-1, keepdims=True)
        out.append(np.ascontiguousarray(s, dtype=np.float32))
    return out


def _target(case, E):
    """A target S(q,t) of the fit's size: a slowly decaying oscillation."""
    t = case["dt"] * case["stride"] * np.arange(1, E + 1)
    return np.exp(-0.3 * t) * (0.9 * np.cos(0.7 * t) + 0.2j * np.sin(0.7 * t))


def _dropin_inputs(case, seed):
    """Host arrays of the fused program's step (kernel_fusion/llg_sqt_fusion.c:370-441):
    spins, A and B of the correlation, the phases q and C in the interleaved
    layout (re rows (i / 4) * 8 + i % 4, im rows + 4, leading dimension 2 N^2)."""
    N, nf = case["N"], case["nfile"]
    M, K = N * N, 3 * nf
    spin = _spins(case, seed).cpu().numpy()
    zero = _spins(case, seed, salt=1).cpu().numpy()
    a = np.ascontiguousarray(spin.transpose(0, 2, 1)).reshape(-1)
    b = np.ascontiguousarray(zero.transpose(1, 0, 2)).reshape(-1)
    i = np.arange(M)
    th = 2.0 * np.pi * (N // 10) / N * ((i // N)[:, None] - (i // N)[None, :]
                                        + (i % N)[:, None] - (i % N)[None, :])
    rows = (i // 4) * 8 + i % 4
    q = np.zeros((M, 2 * M))
    q[:, rows] = np.cos(th).T
    q[:, rows + 4] = -np.sin(th).T
    outer = spin.mean(axis=0) @ zero.mean(axis=0).T
    c = np.zeros((M, 2 * M))
    c[:, rows] = -outer.T * q[:, rows]
    c[:, rows + 4] = -outer.T * q[:, rows + 4]
    return spin, a, b, q, c, M, K


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind in ("series", "grid", "llg", "host"):
        M, nf = case["N"] ** 2, case["nfile"]
        s = _spins(case, seed)
        ctx = asd.Context(_params(case), modes=[case.get("mode", "fp64")])
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        ctx.set_spins_device(s.data_ptr(), as_origin=True)
        if kind == "series":
            st["out"] = torch.zeros(case["evals"], 2, dtype=torch.float64, device="cuda")
        elif kind == "grid":
            st["out"] = torch.zeros(case["evals"], M, 2, dtype=torch.float64, device="cuda")
        if kind != "host":
            st["spins"] = torch.zeros(nf, M, 3, dtype=torch.float64, device="cuda")
        else:
            st["spins"] = s.cpu().pin_memory()
            st["out"] = torch.zeros(case["nsteps"], 2, dtype=torch.float64).pin_memory()
        torch.cuda.synchronize()  # the context has read s
        st["ctx"] = ctx
    elif kind == "loss":
        s = _spins(case, seed)
        ctx = asd.Context(_params(case), modes=["fp64"])
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        ctx.set_spins_device(s.data_ptr(), as_origin=True)
        torch.cuda.synchronize()
        st["ctx"] = ctx
        st["target"] = _target(case, case["nsteps"] // case["stride"])
    elif kind == "batch":
        b = asd.Batch([asd.Lattice.make(n, J1=1.0, alpha=al, dt=case["dt"])
                       for n, _, al in _lattices(case)])
        for l, s in enumerate(_batch_spins(case, seed)):
            b.set_spins(l, s)
        b.autotune(5)
        st["batch"] = b
    else:
        spin, a, b, q, c, M, K = _dropin_inputs(case, seed)
        st.update(spin=spin, a=a, b=b, q=q.reshape(-1), c=c.reshape(-1), M=M, K=K,
                  rk=[np.zeros_like(spin) for _ in range(5)], sum=np.zeros(256))
    return st


# --------------------------------------------------------------------- pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "series":
        ctx, out = st["ctx"], st["out"]
        p = out.data_ptr()
        for e in range(case["evals"]):
            ctx.step(case["stride"])
            ctx.sqt_async(case["mode"], p + 16 * e)
        ctx.get_spins_device(st["spins"].data_ptr())
        return dict(sqt=out, spins=st["spins"])
    if kind == "grid":
        ctx, out = st["ctx"], st["out"]
        p, n = out.data_ptr(), 16 * case["N"] ** 2
        for e in range(case["evals"]):
            ctx.step(case["stride"])
            ctx.sqt_grid_async(case["mode"], p + n * e)
        ctx.get_spins_device(st["spins"].data_ptr())
        return dict(sqt=out, spins=st["spins"])
    if kind == "llg":
        ctx, out = st["ctx"], st["spins"]
        ctx.step(case["nsteps"])
        ctx.get_spins_device(out.data_ptr())
        return out
    if kind == "loss":
        loss, grad, sqt = st["ctx"].loss_grad(case["nsteps"], case["stride"], case["checkpoint"],
                                              st["target"])
        return dict(loss=np.float64(loss), grad=grad, sqt=sqt)
    if kind == "batch":
        b = st["batch"]
        b.run(case["nsteps"])
        return [b.get_spins(l) for l in range(case["count"])]
    if kind == "host":
        ctx, s, out = st["ctx"], st["spins"], st["out"]
        p, o = s.data_ptr(), out.data_ptr()
        for e in range(case["nsteps"]):
            ctx.step_host_async(p, p, case["mode"], o + 16 * e)
        ctx.synchronize()
        return dict(spins=s, sqt=out)
    asd.set_params(case["N"], case["nfile"], case["J1"], case["dt"])
    lib = asd.load()
    ptr = lambda x: ctypes.c_void_p(x.ctypes.data)  # noqa: E731
    lib.runge_kutta(ptr(st["spin"]), *[ptr(x) for x in st["rk"]])
    M, K = st["M"], st["K"]
    st["sum"][:] = 0.0
    asd.fused_dgemm(M, M, K, 1.0 / case["nfile"], st["a"], M, st["b"], K, st["c"], 2 * M, st["q"],
                    st["sum"])
    return dict(cur=st["rk"][0], k1=st["rk"][1], k2=st["rk"][2], k3=st["rk"][3], k4=st["rk"][4],
                c=st["c"], sum=st["sum"][:2].copy())


# --------------------------------------------------------------------- work
def _ops(case):
    """FP64 (batch: FP32) operations of one site-step: the right-hand side and
    dt * f in four stages, the stage combinations, the renormalisation."""
    rhs = 24 + (24 if case["J2"] else 0) + (3 if case["hz"] else 0) + 9 + (18 if case["alpha"] else 0)
    return 4 * (rhs + 3) + 75


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sites = sum(n * n for n, _, _ in _lattices(case))
        return dict(bytes=24.0 * sites, flops=float(sites) * case["nsteps"] * (4 * 54 + 75))
    M, nf = float(case["N"]) ** 2, float(case["nfile"])
    K, state = 3.0 * nf, 24.0 * M * nf
    if kind == "dropin":
        # spins in, the new state and k1..k4 out; A, B, C and q in, C out
        return dict(bytes=6 * state + 2 * 8 * M * K + 3 * 16 * M * M,
                    flops=M * nf * (4 * 33 + 33) + 2 * M * M * K + 4 * M * M)
    if kind == "loss":
        # forward with S at every stride, then per step the stages again, the
        # adjoint of each (about twice a stage's operations) and the gathers
        n = case["nsteps"]
        return dict(bytes=state, flops=M * nf * n * (_ops(case) * 4.0) + M * K * 8.0 * n / case["stride"])
    if kind == "llg":
        return dict(bytes=2 * state, flops=M * nf * case["nsteps"] * _ops(case))
    if kind == "host":
        steps = case["nsteps"]
        per = 6.0 * M * M * K if case["mode"] != "fp64" else 4.0 * M * K
        return dict(bytes=2 * state * steps, flops=steps * (M * nf * _ops(case) + per))
    steps = case["evals"] * case["stride"]
    if case["mode"] != "fp64":  # three products of the split operands
        per = 6.0 * M * M * K
    elif kind == "series":      # one phase-weighted sum per column
        per = 4.0 * M * K
    else:                       # one 2-D transform per column, and the products
        per = K * (5.0 * M * math.log2(M) + 8.0 * M)
    out = 16.0 * case["evals"] * (M if kind == "grid" else 1.0)
    return dict(bytes=3 * state + out, flops=M * nf * _ops(case) * steps + per * case["evals"])


# -------------------------------------------------------------------- exact
def _rhs(s, p):
    """dS/dt on [nfile][N][N][3], p = (J1, J2, alpha, h[3])."""
    J1, J2, al, h = p
    nn = sum(s.roll(d, dims=a) for a in (1, 2) for d in (1, -1))
    H = J1 * nn
    if isinstance(J2, torch.Tensor) or J2 != 0.0:
        H = H + J2 * sum(s.roll((i, j), dims=(1, 2)) for i in (1, -1) for j in (1, -1))
    if h is not None:
        H = H + h
    tau = torch.linalg.cross(H, s)
    if isinstance(al, float) and al == 0.0:
        return tau
    return (tau + al * torch.linalg.cross(s, tau)) / (1.0 + al * al)


def _rk4(s, p, dt, renorm=True):
    k1 = dt * _rhs(s, p)
    k2 = dt * _rhs(s + k1 / 2, p)
    k3 = dt * _rhs(s + k2 / 2, p)
    k4 = dt * _rhs(s + k3, p)
    o = s + k1 / 6 + k2 / 3 + k3 / 3 + k4 / 6
    if not renorm:
        return o, (k1, k2, k3, k4)
    return o / o.norm(dim=-1, keepdim=True)


def _model_of(case, device="cuda", dtype=torch.float64):
    h = torch.tensor([0.0, 0.0, case["hz"]], device=device, dtype=dtype) if case["hz"] else None
    return (case["J1"], case["J2"], case["alpha"], h)


def _lat(case, s):
    return s.reshape(case["nfile"], case["N"], case["N"], 3)


def _phase(N):
    i = torch.arange(N * N, device="cuda", dtype=torch.float64)
    th = 2.0 * math.pi * (N // 10) / N * (torch.div(i, N, rounding_mode="floor") + i % N)
    return torch.polar(torch.ones_like(th), -th)


def _sums(s, u):
    """sum_i u_i s_i per replica and component, [nfile][3] complex."""
    return torch.complex(torch.einsum("i,fic->fc", u.real, s), torch.einsum("i,fic->fc", u.imag, s))


def _sqt(case, s, zero):
    N, nf = case["N"], case["nfile"]
    u = _phase(N)
    F = _sums(s.reshape(nf, N * N, 3), u)
    G = _sums(zero.reshape(nf, N * N, 3), u.conj())
    return (F * (G - G.mean(dim=0, keepdim=True))).sum() / (N * N * nf)


def _grid(case, s, zero):
    """S(q,t) at every q = 2 pi (a, b) / N."""
    N, nf = case["N"], case["nfile"]
    acc = torch.zeros(N, N, device="cuda", dtype=torch.complex128)
    m, z = s.mean(dim=0), zero.mean(dim=0)
    for f0 in range(0, nf, 64):
        A = torch.fft.fft2(_lat(case, s)[f0:f0 + 64] - m.reshape(1, N, N, 3), dim=(1, 2))
        B = torch.fft.fft2(_lat(case, zero)[f0:f0 + 64] - z.reshape(1, N, N, 3), dim=(1, 2))
        acc += (A * B.conj()).sum(dim=(0, 3))
    return torch.view_as_real(acc.reshape(-1)) / (N * N * nf)


def _exact_loss(case, seed):
    from torch.utils.checkpoint import checkpoint

    E = case["nsteps"] // case["stride"]
    s0 = _lat(case, _spins(case, seed))
    v = torch.tensor([case["J1"], case["J2"], case["alpha"], 0.0, 0.0, case["hz"]], device="cuda",
                     dtype=torch.float64, requires_grad=True)
    step = lambda s, w: _rk4(s, (w[0], w[1], w[2], w[3:6]), case["dt"])  # noqa: E731
    tgt = torch.from_numpy(_target(case, E)).cuda()
    s, L, vals = s0, 0.0, []
    for n in range(1, case["nsteps"] + 1):
        s = checkpoint(step, s, v, use_reentrant=False)
        if n % case["stride"] == 0 and n // case["stride"] <= E:
            S = _sqt(case, s, s0)
            d = torch.view_as_real(S - tgt[n // case["stride"] - 1])
            L = L + (d * d).sum() / E
            vals.append(S.detach())
    L.backward()
    return dict(loss=L.detach(), grad=v.grad, sqt=torch.stack(vals))


def _exact_batch(case, seed):
    lats, spins = _lattices(case), _batch_spins(case, seed)
    out = [None] * len(lats)
    for n in sorted({l[0] for l in lats}):
        at = [i for i, l in enumerate(lats) if l[0] == n]
        s = torch.stack([torch.from_numpy(spins[i]).cuda().double() for i in at]).reshape(-1, n, n, 3)
        al = torch.tensor([lats[i][2] for i in at], device="cuda",
                          dtype=torch.float32).double().reshape(-1, 1, 1, 1)
        for _ in range(case["nsteps"]):
            s = _rk4(s, (1.0, 0.0, al, None), float(np.float32(case["dt"])))
        for k, i in enumerate(at):
            out[i] = s[k].reshape(-1, 3)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "loss":
        return _exact_loss(case, seed)
    p = _model_of(case)
    if kind == "dropin":
        spin, a, b, q, c, M, K = _dropin_inputs(case, seed)
        cur, k = _rk4(_lat(case, torch.from_numpy(spin).cuda()), p, case["dt"], renorm=False)
        flat = lambda t: t.reshape(case["nfile"], M, 3)  # noqa: E731
        A = torch.from_numpy(a).cuda().reshape(K, M).T
        B = torch.from_numpy(b).cuda().reshape(M, K).T
        P = (A @ B / case["nfile"]).T
        rows = torch.from_numpy((np.arange(M) // 4) * 8 + np.arange(M) % 4).cuda()
        Q, Cm = torch.from_numpy(q).cuda(), torch.from_numpy(c).cuda()
        Cm[:, rows] += Q[:, rows] * P
        Cm[:, rows + 4] += Q[:, rows + 4] * P
        return dict(cur=flat(cur), k1=flat(k[0]), k2=flat(k[1]), k3=flat(k[2]), k4=flat(k[3]),
                    c=Cm.reshape(-1), sum=torch.stack([Cm[:, rows].sum(), Cm[:, rows + 4].sum()]))
    zero = _spins(case, seed)
    s = _lat(case, zero)
    if kind == "llg":
        for _ in range(case["nsteps"]):
            s = _rk4(s, p, case["dt"])
        return s.reshape(case["nfile"], -1, 3)
    if kind == "host":
        vals = []
        for _ in range(case["nsteps"]):
            s = _rk4(s, p, case["dt"])
            vals.append(torch.view_as_real(_sqt(case, s, zero)))
        return dict(spins=s.reshape(case["nfile"], -1, 3), sqt=torch.stack(vals))
    vals = []
    for _ in range(case["evals"]):
        for _ in range(case["stride"]):
            s = _rk4(s, p, case["dt"])
        vals.append(_grid(case, s, zero) if kind == "grid"
                    else torch.view_as_real(_sqt(case, s, zero)))
    return dict(sqt=torch.stack(vals), spins=s.reshape(case["nfile"], -1, 3))
