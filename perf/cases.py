"""The performance cases of the contour-advection library.

Each case is a piece of work a program gives the library through its public
entry points (include/hydra_casl.h, hydra_b200/casl.py):

``window``     a saved state is loaded, advanced by a few time steps and read
               back: a restart, or the stretch between two outputs.  A step is
               what the library is for; the kind spans the grids it accepts
               (32^2 to 2048^2) and the options that runs switch on (surgery
               every step or when the twist asks for it, QG on a beta-plane,
               friction and thermal damping, the FP32 inversion, the learned
               closure).
``recontour``  new contours from contours plus a residual field, which a run
               does every 20 regularisations; without contours in the state it
               is how a run starts.
``ensemble``   members of uneven size from their initial fields through some
               steps, in one handle.
``con2grid``   contours to gridded PV on arrays the caller owns on the GPU.
``invert``     velocity and streamfunction of a spectral PV field, for a host
               program that keeps its own fields.
``network``    the closure's network on a batch of host data, forward and
               gradient, as a training loop outside the library calls it.

Host buffers are pinned, as a program that moves its state every few steps
keeps them.
"""
from __future__ import annotations

import ctypes as C
import os

import numpy as np
import torch

from hydra_b200 import casl
from hydra_b200.casl import NET_IN, NET_OUT, CaslEnsemble, CaslGPU, CaslNet
from hydra_b200.synthetic import ensemble_member_params, random_pv

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(casl.__file__)), "closure_512.npz")
PLAIN = dict(kd=0.0, beta=0.0, rekman=0.0, rtherm=0.0, every=True, fp32=False, closure=False)


def listed():
    return [
        # A small run (the size of a quick look or a parameter scan): latency
        # and launches are all of it.
        dict(name="window 64", kind="window", n=64, k0=4.0, levels=20, steps=16, **PLAIN),
        # The plain workload of a single CPU-sized simulation, 40 levels.
        dict(name="window 256", kind="window", n=256, k0=6.0, levels=40, steps=16, **PLAIN),
        # QG turbulence on a beta-plane with Ekman and thermal damping; surgery
        # only when the accumulated twist asks for it, as the reference runs.
        dict(name="window 512 beta", kind="window", n=512, k0=12.0, levels=80, steps=16, kd=2.5,
             beta=10.0, rekman=0.1, rtherm=0.05, every=False, fp32=False, closure=False),
        # The learned closure in every stage of the step.
        dict(name="window 512 closure", kind="window", n=512, k0=12.0, levels=80, steps=10,
             **dict(PLAIN, closure=True)),
        # The benchmark's workload: 1024^2, 80 levels, surgery every step.
        dict(name="window 1024", kind="window", n=1024, k0=16.0, levels=80, steps=10, **PLAIN),
        # The largest grid: beta-plane QG with the FP32 inversion.
        dict(name="window 2048 fp32", kind="window", n=2048, k0=12.0, levels=48, steps=5,
             **dict(PLAIN, kd=2.5, beta=10.0, fp32=True)),
        # The recontouring of the benchmark's workload.
        dict(name="recontour 1024", kind="recontour", n=1024, k0=16.0, levels=80, beta=0.0,
             contours=True),
        # A member-sized beta-plane run's start: contours from its first field.
        dict(name="recontour 256 beta", kind="recontour", n=256, k0=6.0, levels=40, beta=10.0,
             contours=False),
        # Members of uneven size from fields to a short forecast.
        dict(name="ensemble 48x256", kind="ensemble", n=256, members=48, steps=10),
        # Gridded PV for an analysis that holds its contours on the GPU.
        dict(name="con2grid 128", kind="con2grid", n=128, k0=5.0, levels=30),
        # One inversion for a host program with its own spectral fields.
        dict(name="invert 1024", kind="invert", n=1024, kd=2.5),
        # One training sample of the closure's network outside the library.
        dict(name="network 512", kind="network", n=512),
    ]


def draw(rng):
    kind = rng.choice(["window"] * 5 + ["recontour"] * 2 + ["ensemble", "con2grid", "invert", "network"])
    beta = rng.choice([0.0, 10.0])
    if kind == "window":
        n = rng.choice([32, 64, 128, 256, 512, 1024, 2048])
        k0, levels = _contouring(rng, n, beta)
        closure = n in (128, 256, 512, 1024) and rng.random() < 0.2
        return dict(kind=kind, n=n, k0=k0, levels=levels, steps=rng.randint(3, 8), kd=rng.choice([0.0, 1.0, 2.5]), beta=beta,
                    rekman=rng.choice([0.0, 0.1]), rtherm=rng.choice([0.0, 0.05]),
                    every=rng.random() < 0.7, fp32=n >= 128 and rng.random() < 0.3, closure=closure)
    if kind == "recontour":
        n = rng.choice([32, 64, 128, 256, 512, 1024])
        k0, levels = _contouring(rng, n, beta)
        return dict(kind=kind, n=n, k0=k0, levels=levels, beta=beta, contours=rng.random() < 0.6)
    if kind == "ensemble":
        n = rng.choice([64, 128, 256])
        return dict(kind=kind, n=n, members=rng.randint(3, 40), steps=rng.randint(3, 10))
    if kind == "con2grid":
        n = rng.choice([32, 64, 128, 256])
        k0, levels = _contouring(rng, n, 0.0)
        return dict(kind=kind, n=n, k0=k0, levels=levels)
    if kind == "invert":
        return dict(kind=kind, n=rng.choice([32, 64, 128, 256, 512, 1024, 2048]),
                    kd=round(rng.uniform(0.0, 5.0), 2))
    return dict(kind=kind, n=128 * rng.randint(1, 6))


def _k0_most(n):
    return min(24.0, 3.0 + n / 64.0)


def _contouring(rng, n, beta):
    """A spectral peak the grid resolves and a number of PV jumps; on the
    largest grids no more of both than the listed cases have."""
    k0 = round(rng.uniform(3.0, _k0_most(n)), 2)
    levels = rng.randint(12, 96)
    most = {1024: 1500, 2048: 1152}.get(n)
    if most:
        levels = min(levels, int(most / k0 / (2 if beta else 1)))
    return k0, levels


def _nodes(case):
    """About how many nodes the case's first contours have.  On a beta-plane
    the jump is set by beta Ly, about half the field's range."""
    n = case["n"]
    size = 1000.0 * (n / 1024.0) ** 0.75
    if case["kind"] == "ensemble":
        return case["members"] * 320.0 * size
    return case["k0"] * case["levels"] * size * (2.0 if case.get("beta") else 1.0)


def work(case):
    """A step reads and writes the nodes (x, y, successor) and the two spectral
    fields once; its operations are the 37 2-D transforms and the four
    stages' node updates.  A recontouring reads its field and contours and
    writes contours; its operations are the evaluation of the 16x field."""
    kind, n = case["kind"], case["n"]
    nn = float(n) * n
    fft = 2.5 * nn * 2.0 * np.log2(n)
    if kind in ("window", "ensemble"):
        k, m = case["steps"], case.get("members", 1)
        pts = _nodes(case)
        flops = k * (m * 37 * fft + pts * 4 * 60)
        if case.get("closure"):
            flops += k * 4 * _net_flops(n)
        start = m * 256 * nn * 10 if kind == "ensemble" else 0.0
        return {"bytes": k * 2 * (20 * pts + 16 * m * nn), "flops": flops + start}
    if kind == "recontour":
        return {"bytes": 8 * nn + (2 if case["contours"] else 1) * 20 * _nodes(case), "flops": 256 * nn * 10}
    if kind == "con2grid":
        return {"bytes": 8 * nn + 20 * _nodes(case), "flops": 40 * _nodes(case)}
    if kind == "invert":
        return {"bytes": 5 * 8 * nn, "flops": 2 * fft + 5 * nn}
    return {"bytes": 4 * nn * (NET_IN + 2 * NET_OUT), "flops": 3 * _net_flops(n)}


def _net_flops(n):
    return 2.0 * 25 * n * n * (NET_IN * 16 + 16 * 16 + 16 * 16 + 16 * NET_OUT)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _pinned(count, dtype):
    return torch.zeros(int(count), dtype=dtype).pin_memory().numpy()


def _pin(a):
    dtype = {"f8": torch.float64, "i4": torch.int32, "f4": torch.float32}[a.dtype.str[1:]]
    p = _pinned(a.size, dtype)
    p[:] = a.reshape(-1)
    return p.reshape(a.shape)


def _ptr(a):
    t = {"f8": C.c_double, "i4": C.c_int, "f4": C.c_float}[a.dtype.str[1:]]
    return a.ctypes.data_as(C.POINTER(t))


class Buffers:
    """Pinned host arrays of the run's capacity for a state to be read back
    into (zero beyond its counts)."""

    def __init__(self, n, nodes, contours, fields=True):
        self.xy = [_pinned(nodes, torch.float64) for _ in range(2)]
        self.nextq = _pinned(nodes, torch.int32)
        self.cont = [_pinned(contours, torch.int32) for _ in range(4)]  # indq npq i1q i2q
        self.fields = [_pinned(n * n, torch.float64).reshape(n, n) for _ in range(2 if fields else 0)]

    def read(self, g):
        nq, npt, qj = g.counts()
        g._check(g.lib.casl_get_contours(g.h, _ptr(self.xy[0]), _ptr(self.xy[1]), _ptr(self.nextq),
                                         *[_ptr(a) for a in self.cont]), "casl_get_contours")
        out = dict(nq=nq, nptq=npt, qjump=qj, xq=self.xy[0], yq=self.xy[1], nextq=self.nextq)
        out.update(zip(("indq", "npq", "i1q", "i2q"), self.cont))
        for name, a in zip(("qs", "qd"), self.fields):
            which = casl.FIELDS[name]
            g._check(g.lib.casl_get_field(g.h, which, _ptr(a)), "casl_get_field")
            out[name] = a
        return out


def _capacity(case):
    """Node capacity: a few times what the first contours have."""
    return int(max(1 << 17, 4 * _nodes(case)))


def _simulation(case, **more):
    npm = _capacity(case)
    kw = dict(ncontq=case["levels"], kd=case.get("kd", 0.0), beta=case.get("beta", 0.0),
              rekman=case.get("rekman", 0.0), rtherm=case.get("rtherm", 0.0), dtmax=0.05, npm=npm,
              nm=npm // 8)
    kw.update(more)
    return CaslGPU(case["n"], **kw)


def _pin_contours(c):
    return {k: (_pin(v) if isinstance(v, np.ndarray) else v) for k, v in c.items()}


def _network(n, seed):
    d = np.load(WEIGHTS)
    net = CaslNet(n)
    net.set_params(d["params"], float(d["qscale"]), float(d["uscale"]))
    return net


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "ensemble":
        seeds = [seed * 1000 + m for m in range(case["members"])]
        params = [ensemble_member_params(s) for s in seeds]
        npm = _capacity(case)
        g = CaslEnsemble(n, case["members"], npm=npm, nm=npm // 8, dtmax=0.05)
        most = _k0_most(n)
        return dict(case=case, g=g, fields=[random_pv(n, min(p[0], most), s) for s, p in zip(seeds, params)],
                    levels=[p[1] for p in params], out=Buffers(n, npm, npm // 8, fields=False))
    if kind == "invert":
        rng = np.random.default_rng(seed)
        k = np.minimum(np.arange(n), n - np.arange(n)).astype(np.float64)
        K = np.hypot(k[:, None], k[None, :])
        q = rng.standard_normal((n, n)) * n / (1.0 + K) ** 1.5
        q[0, 0] = 0.0
        g = CaslGPU(n, kd=case["kd"], npm=1 << 16, nm=1 << 12)
        out = [_pinned(n * n, torch.float64).reshape(n, n) for _ in range(3)]
        return dict(case=case, g=g, q=_pin(q), out=out)
    if kind == "network":
        x, dy = _network_inputs(n, seed)
        net = _network(n, seed)
        return dict(case=case, net=net, x=_pin(x), dy=_pin(dy),
                    y=_pinned(NET_OUT * n * n, torch.float32).reshape(NET_OUT, n, n),
                    grad=_pinned(net.count, torch.float32))
    q0 = random_pv(n, case["k0"], seed)
    if kind == "con2grid":
        g = _simulation(case)
        g.initialise(q0)
        c = g.contours()
        g.close()
        dev = {k: torch.from_numpy(c[k]).cuda() for k in ("xq", "yq", "nextq")}
        return dict(case=case, lib=g.lib, qjump=c["qjump"], nptq=c["nptq"], **dev,
                    qc=torch.empty(n, n, dtype=torch.float64, device="cuda"))
    if kind == "recontour":
        # the residual a run recontours with is a few per cent of a jump
        g = _simulation(case)
        state = dict(case=case, g=g, out=Buffers(n, _capacity(case), _capacity(case) // 8, fields=False))
        if not case["contours"]:
            return dict(state, q=_pin(q0), start=None)
        g.initialise(q0)
        res = random_pv(n, min(case["k0"], n / 8.0), seed + 1, rms=0.1 * g.counts()[2], power=1.0)
        return dict(state, q=_pin(res), start=_pin_contours(g.contours()))
    # the saved state comes from a run of its own
    first = _simulation(case)
    first.initialise(q0)
    start, qs, qd = _pin_contours(first.contours()), _pin(first.field("qs")), _pin(first.field("qd"))
    first.close()
    g = _simulation(case, force_surgery=int(case["every"]))
    if case["fp32"]:
        g.set_precision(1)
    state = dict(case=case, g=g, start=start, qs=qs, qd=qd,
                 out=Buffers(n, _capacity(case), _capacity(case) // 8))
    if case["closure"]:
        state["net"] = _network(n, seed)
        g.closure_attach(state["net"])
    return state


def _network_inputs(n, seed):
    """Smooth fields of unit size for PV and velocity, rough ones for the
    sub-cell levels, and an output gradient."""
    x = np.empty((NET_IN, n, n), np.float32)
    m = 1 << (n - 1).bit_length()
    for c in range(3):
        x[c] = random_pv(m, 6.0, seed + c, rms=1.0)[:n, :n]
    rng = np.random.default_rng(seed)
    x[3:] = 0.1 * rng.standard_normal((NET_IN - 3, n, n))
    return x, rng.standard_normal((NET_OUT, n, n)).astype(np.float32)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind, n = case["kind"], case["n"]
    if kind == "window":
        g = s["g"]
        g.set_contours(s["start"])
        g.set_field("qs", s["qs"])
        g.set_field("qd", s["qd"])
        g.set_scalar("t", 0.0)
        # with surgery on demand: a state about to ask for it
        g.set_scalar("twist", 0.0 if case["every"] else 2.0)
        g.set_scalar("ireg", 0)
        g.step(case["steps"])
        return s["out"].read(g)
    if kind == "recontour":
        g = s["g"]
        if s["start"] is None:
            g.initialise(s["q"])
        else:
            g.set_contours(s["start"])
            g.recontour(s["q"])
        return s["out"].read(g)
    if kind == "ensemble":
        g = s["g"]
        g.initialise_members(s["fields"], s["levels"])
        g.step(case["steps"])
        return s["out"].read(g)
    if kind == "con2grid":
        two_pi = 2.0 * np.pi
        stream = torch.cuda.current_stream().cuda_stream
        rc = s["lib"].casl_con2grid_noalloc(n, two_pi, two_pi, s["nptq"], s["qjump"],
                                            s["xq"].data_ptr(), s["yq"].data_ptr(),
                                            s["nextq"].data_ptr(), s["qc"].data_ptr(), stream)
        if rc:
            raise RuntimeError(f"casl_con2grid_noalloc: {rc}")
        return s["qc"]
    if kind == "invert":
        g = s["g"]
        g._check(g.lib.casl_main_invert(g.h, _ptr(s["q"]), *[_ptr(a) for a in s["out"]]), "casl_main_invert")
        return s["out"]
    net = s["net"]
    net._check(net.lib.casl_net_forward(net.h, _ptr(s["x"]), _ptr(s["y"])), "casl_net_forward")
    net._check(net.lib.casl_net_backward(net.h, _ptr(s["dy"]), _ptr(s["grad"])), "casl_net_backward")
    return s["y"], s["grad"]


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "con2grid":
        return _exact_con2grid(case, seed)
    if kind == "invert":
        return _exact_invert(case, seed)
    if kind == "network":
        return _exact_network(case, seed)
    return None  # surgery and renode decide node by node: minutes in numpy


def _exact_con2grid(case, seed):
    s = prepare(case, seed)
    x, y = s["xq"].cpu().numpy(), s["yq"].cpu().numpy()
    ia = s["nextq"].cpu().numpy().astype(np.int64) - 1
    n, ell = case["n"], 2.0 * np.pi
    nf, half = 4 * n, np.pi
    gl = ell / nf
    ixc = np.trunc((nf / ell) * (x + half)).astype(np.int64)
    dx = x[ia] - x
    dx -= ell * np.trunc(dx / half)
    yy = y[ia] - y
    dy = yy - ell * np.trunc(yy / half)
    jump = np.zeros((nf, nf), np.int64)  # [column, row]
    d = ixc[ia] - ixc
    ncr = d - nf * np.trunc(2.0 * d / nf).astype(np.int64)
    for k in range(int(np.abs(ncr).max())):
        i = np.nonzero(np.abs(ncr) > k)[0]
        sg = np.sign(ncr[i])
        col = (ixc[i] + (sg > 0) + k * sg) % nf
        x2 = -half + gl * col - x[i]
        p = (x2 - ell * np.trunc(x2 / half)) / dx[i]
        y2 = y[i] + p * dy[i]
        row = 1 + np.trunc((nf / ell) * (y2 - ell * np.trunc(y2 / half) + half)).astype(np.int64)
        ok = (row >= 1) & (row < nf)
        np.add.at(jump, (col[ok], row[ok]), np.where(dx[i] >= 0, 1, -1)[ok])
    i = np.nonzero(np.abs(yy) > half)[0]
    sg = np.where(dy[i] >= 0, 1.0, -1.0)
    p = -(y[i] - half * sg) / (dy[i] + 1.0e-12)
    col = np.trunc((nf / ell) * np.fmod(ell + half + x[i] + p * dx[i], ell)).astype(np.int64) % nf
    bottom = np.zeros(nf, np.int64)
    np.add.at(bottom, col, -sg.astype(np.int64))
    jump[:, 0] = np.cumsum(bottom) - bottom
    level = np.cumsum(jump, axis=1).astype(np.float64)
    for axis in (0, 1):
        for _ in range(2):
            level = 0.5 * level + 0.25 * (np.roll(level, 1, axis) + np.roll(level, -1, axis))
            level = np.take(level, np.arange(0, level.shape[axis], 2), axis)
    return s["qjump"] * (level - level.mean())


def _hermitian_inverse(s, axis):
    s = np.moveaxis(s, axis, 0)
    n = s.shape[0]
    F = np.zeros((n // 2 + 1,) + s.shape[1:], np.complex128)
    F.real = s[: n // 2 + 1]
    F.imag[1:n // 2] = s[n - np.arange(1, n // 2)]
    return np.moveaxis(np.fft.irfft(F, n, axis=0) * np.sqrt(n), 0, axis)


def _exact_invert(case, seed):
    n, kd = case["n"], case["kd"]
    q = np.array(prepare(case, seed)["q"])  # [ky, kx]
    k = np.arange(n)
    k = np.minimum(k, n - k).astype(np.float64)
    k2 = k[:, None] ** 2 + k[None, :] ** 2 + kd * kd
    k2[0, 0] = 1.0
    pp = -q / k2
    pp[0, 0] = 0.0
    fac = np.where(np.arange(n) < n // 2, -1.0, 1.0) * k * np.exp(-36.0 * (2.0 * k / n) ** 36)
    fac[n // 2] = 0.0
    back = (-np.arange(n)) % n
    vx = fac[None, :] * pp[:, back]
    uy = fac[:, None] * pp[back, :]
    phys = [_hermitian_inverse(_hermitian_inverse(a, 0), 1).T for a in (uy, vx)]
    return [-phys[0], phys[1], pp]


def _exact_network(case, seed):
    n = case["n"]
    x, dy = (torch.from_numpy(a).cuda().double() for a in _network_inputs(n, seed))
    flat = torch.from_numpy(np.load(WEIGHTS)["params"]).cuda().double().requires_grad_(True)
    sizes = [(NET_IN, 16), (16, 16), (16, 16), (16, NET_OUT)]
    a, at = x, 0
    for layer, (ci, co) in enumerate(sizes):
        w = flat[at:at + co * ci * 25].reshape(co, ci, 5, 5)
        at += co * ci * 25
        b = flat[at:at + co]
        at += co
        z = b[:, None, None].expand(co, n, n)
        for ky in range(5):
            for kx in range(5):
                z = z + torch.einsum("oi,ihw->ohw", w[:, :, ky, kx], torch.roll(a, (2 - ky, 2 - kx), (1, 2)))
        a = torch.nn.functional.gelu(z) if layer < 3 else z
    a.backward(dy)
    return a.detach(), flat.grad.detach()
