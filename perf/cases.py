"""Performance cases of the Gross-Pitaevskii stepper, through its public entry
points: time stepping of one solve (fixed step, adaptive step, imaginary time),
batches of solves, the diagnostics a run writes at its save points, the norm
of a caller-owned array and initial states made on the device.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program has in hand before the call
    run(state)           one pass through the public entry points
    work(case)           bytes and operations a pass cannot do without
    exact(case, seed)    the outputs in 64 bits by plain torch, without this package

A state of a stepping case lives on the GPU in a caller's tensor: a pass hands
it over (gpe_set_state_device), steps it, and takes the result back
(gpe_get_state_device), so every pass starts from the same inputs.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

from gpe_b200 import _lib as L
from gpe_b200 import ic
from gpe_b200.pool import Pool
from gpe_b200.solver import RunParams, Solver

PI = 3.1415926535897932384626433832795
# the sites x steps a drawn case may have (those of the largest listed one)
MOST = 256 ** 3 * 20


# ---------------------------------------------------------------------------
# the cases


def _steps(name, n, steps, **kw):
    c = dict(name=name, kind="steps", nx=n[0], ny=n[1], nz=n[2], steps=steps, scheme="rk4", eqn=4, bcs=1, order=4,
             storage="c128", tau=0.01, dx=0.5, Urhs=0.0, diss=0.0, mu=1.0, om=0.0, gamma=0.0, ic="turbulence")
    c.update(kw)
    return c


def listed():
    return [
        # the headline workload: turbulence in a periodic box, many steps between outputs
        _steps("rk4_256_c128", (256, 256, 256), 20, eqn=2, tau=0.005),
        # the same box with complex64 storage, the other storage a run can choose
        _steps("rk4_256_c64", (256, 256, 256), 20, eqn=2, tau=0.005, storage="c64"),
        # a vortex ring in a small reflecting box, second order: the reference's introductory run, one
        # 100-step chunk of the time loop
        _steps("rk4_ring_64_c128", (64, 64, 64), 100, bcs=2, order=2, ic="ring"),
        # the smallest call: a quick look at a tiny box, where launches and latency are all there is
        _steps("rk4_tiny_c128", (32, 28, 24), 10, bcs=2, ic="ring"),
        # flow past the frame of a moving ring with a dissipative sponge at the walls; odd and ragged sizes
        _steps("rk4_sponge_odd_c128", (131, 97, 115), 40, eqn=1, bcs=2, Urhs=0.2, diss=0.1, ic="ring"),
        # a trapped, damped condensate with complex64 storage on odd sizes
        _steps("rk4_trap_odd_c64", (75, 150, 203), 40, bcs=2, storage="c64", om=0.06, gamma=0.02, mu=4.0, ic="trap"),
        # the adaptive scheme on the trapped condensate with a vortex line
        _steps("rk45_trap_c128", (192, 192, 384), 3, scheme="rk45", bcs=2, om=0.05, gamma=0.05, mu=10.0, dx=0.25,
               ic="trap"),
        # relaxation to the ground state: imaginary time, the norm taken and put back after every step
        _steps("relax_128_c128", (128, 128, 128), 10, kind="relax", bcs=2, om=0.1, mu=8.0, dx=0.25, tau=0.002,
               ic="trap"),
        # a parameter study: uneven solves of both orders, boundaries, storages and schemes in one pool
        dict(name="batch_mix", kind="batch", solves=16, steps=40, low=32, high=160, study=7),
        # a save point: norm, energy, condensate fraction and spectra of the current state
        _steps("save_point_256_c128", (256, 256, 256), 1, kind="save", eqn=2),
        # the norm of a framework's own array between its steps
        dict(name="norm_192_c128", kind="norm", nx=192, ny=192, nz=384, dx=0.25, storage="c128"),
        # a served request's initial state made on the device: trapped condensate with a vortex line
        dict(name="initial_state_192_c128", kind="initial", nx=192, ny=192, nz=384, dx=0.25, om=0.05, mu=10.0,
             bcs=2, storage="c128", factors="fermi,line_pade"),
    ]


def _size(rng, low, high):
    """A grid extent, log-uniform; every other one a multiple of 16 where that is possible, as users choose them."""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    if rng.random() < 0.5 and n >= 24:
        n = (n + 8) // 16 * 16
    return max(low, min(high, n))


def draw(rng: random.Random):
    kind = rng.choices(["steps", "rk45", "relax", "batch", "save", "norm", "initial"],
                       [45, 14, 10, 9, 9, 7, 6])[0]
    n = tuple(_size(rng, 24, 288) for _ in range(3))
    while n[0] * n[1] * n[2] > 256 ** 3:
        n = tuple(_size(rng, 24, 288) for _ in range(3))
    sites = n[0] * n[1] * n[2]
    storage = rng.choice(["c128", "c64"])
    order, bcs = rng.choice([2, 4, 4]), rng.choice([1, 2])
    if kind == "steps":
        c = _steps("", n, max(1, min(rng.choice([1, 5, 20, 100]), MOST // (2 * sites))),
                   scheme=rng.choice(["rk4"] * 6 + ["rk2", "euler"]), eqn=rng.choice([1, 2, 4, 4]), bcs=bcs,
                   order=order, storage=storage, tau=rng.choice([0.002, 0.005, 0.01]))
        if c["scheme"] == "euler":
            c.update(tau=0.0005)
        if c["eqn"] == 4:
            c["ic"] = rng.choice(["trap", "ring"]) if bcs == 2 else "turbulence"
            if c["ic"] == "trap":
                c.update(om=0.06, mu=4.0, gamma=rng.choice([0.0, 0.02]))
        else:
            c["ic"] = "ring" if bcs == 2 else "turbulence"
            c["Urhs"] = rng.choice([0.0, 0.2])
            c["diss"] = rng.choice([0.0, 0.1]) if c["eqn"] == 1 else 0.0
    elif kind == "rk45":
        c = _steps("", n, max(1, min(rng.choice([2, 4, 8]), MOST // (6 * sites))), scheme="rk45", bcs=2, order=order,
                   storage=storage, om=0.05, gamma=0.05, mu=10.0, dx=0.25, ic="trap")
    elif kind == "relax":
        c = _steps("", n, max(1, min(10, MOST // (3 * sites))), kind="relax", bcs=2, order=order, om=0.1, mu=8.0,
                   storage=storage, dx=0.25, tau=0.002, ic="trap")
    elif kind == "batch":
        c = dict(kind="batch", solves=rng.choice([4, 9, 16, 24]), steps=rng.choice([10, 20, 40]), low=24,
                 high=rng.choice([64, 96, 128]), study=rng.randrange(1 << 20))
    elif kind == "save":
        c = _steps("", n, 1, kind="save", eqn=2, bcs=bcs, order=order, storage=storage)
    elif kind == "norm":
        c = dict(kind="norm", nx=n[0], ny=n[1], nz=n[2], dx=0.25, storage=storage)
    else:
        c = dict(kind="initial", nx=n[0], ny=n[1], nz=n[2], dx=0.25, om=0.05, mu=10.0, bcs=bcs, storage=storage,
                 factors=rng.choice(["fermi,line_pade", "ring", "fermi,line"]))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs


def _rp(c):
    h = [0.5 * c["dx"] * (c[a] - 1) for a in ("nx", "ny", "nz")]
    return RunParams(nx=c["nx"], ny=c["ny"], nz=c["nz"], xr=h[0], yr=h[1], zr=h[2], tau=c["tau"],
                     scheme=c["scheme"], eqn_to_solve=c["eqn"], bcs=c["bcs"], order=c["order"],
                     real_time=c["kind"] != "relax", Urhs=c["Urhs"], diss_amp=c["diss"], g=1.0, mu=c["mu"],
                     nn=_norm_goal(c) if c["kind"] == "relax" else 1.0, omx=c["om"], omy=c["om"], omz=c["om"],
                     gamma=c["gamma"], storage=c["storage"])


def _norm_goal(c):
    """The particle number a relaxation holds: that of a density of one."""
    return float(c["nx"] * c["ny"] * c["nz"]) * c["dx"] ** 3


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _axes(c, dev):
    """x, y, z of the grid, shaped to broadcast over (nz, ny, nx)."""
    out = []
    for ax, n in enumerate((c["nx"], c["ny"], c["nz"])):
        h = 0.5 * c["dx"] * (n - 1)
        q = -h + torch.arange(n, dtype=torch.float64, device=dev) * ((2.0 * h) / (n - 1))
        out.append(q.reshape([-1 if d == 2 - ax else 1 for d in range(3)]))
    return out


def _turbulence(c, seed, dev):
    """Random phases at |k| < 1.5, mean density one (the periodic box's usual start)."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    shape = (c["nz"], c["ny"], c["nx"])
    k = [2.0 * PI * torch.fft.fftfreq(n, d=c["dx"], dtype=torch.float64, device=dev) for n in shape]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    at = torch.nonzero(k2.reshape(-1) < 1.5 ** 2).reshape(-1)
    th = 2.0 * PI * torch.rand(at.numel(), generator=g, dtype=torch.float64).to(dev)
    spec = torch.zeros(k2.numel(), dtype=torch.complex128, device=dev)
    spec[at] = torch.polar(torch.ones_like(th), th)
    psi = torch.fft.ifftn(spec.reshape(shape))
    return psi / torch.sqrt((psi.real ** 2 + psi.imag ** 2).mean())


def _core(r):
    """The Pade vortex core R(r)/r."""
    r2 = r * r
    return torch.sqrt((0.3437 + 0.0286 * r2) / ((1.0 + 0.3333 * r2) + 0.0286 * r2 * r2))


def _ring(c, seed, dev):
    """A vortex ring, off centre by a seeded amount."""
    r = random.Random(seed)
    x, y, z = _axes(c, dev)
    h = 0.5 * c["dx"] * (min(c["nx"], c["ny"], c["nz"]) - 1)
    r0, x0, y0, z0 = h * r.uniform(0.3, 0.5), h * r.uniform(-0.2, 0.2), h * r.uniform(-0.2, 0.2), h * r.uniform(-.2, .2)
    s = torch.sqrt((x - x0) ** 2 + (y - y0) ** 2)
    w = z - z0
    psi = torch.ones((c["nz"], c["ny"], c["nx"]), dtype=torch.complex128, device=dev)
    for b, sign in ((s + r0, 1.0), (s - r0, -1.0)):
        q = _core(torch.sqrt(w * w + b * b))
        psi = psi * torch.complex(q * w, sign * q * b)
    return psi


def _trapped(c, seed, dev):
    """A trapped Thomas-Fermi cloud, everywhere above zero, with a seeded vortex line and a little sound."""
    r = random.Random(seed)
    x, y, z = _axes(c, dev)
    h = 0.5 * c["dx"] * (min(c["nx"], c["ny"]) - 1)
    x0, y0 = h * r.uniform(-0.2, 0.2), h * r.uniform(-0.2, 0.2)
    v = 0.5 * (c["om"] ** 2 * (x * x + y * y + z * z))
    f = torch.sqrt(torch.clamp(c["mu"] - v, min=0.2))
    d = torch.sqrt((x - x0) ** 2 + (y - y0) ** 2)
    line = _core(d)
    wave = 1.0 + 0.02 * torch.sin(0.7 * x + r.uniform(0, 6)) * torch.cos(0.6 * z + r.uniform(0, 6))
    return torch.complex(f * line * (x - x0) * wave, f * line * (y - y0) * wave)


def _state(c, seed, dev):
    return {"turbulence": _turbulence, "ring": _ring, "trap": _trapped}[c["ic"]](c, seed, dev)


def _dtypes(storage):
    """(torch dtype, GPE dtype code) of a state with this storage."""
    return (torch.complex64, L.GPE_C64) if storage == "c64" else (torch.complex128, L.GPE_C128)


def _study(c):
    """The parameter study's solves: uneven cubes, as the batched benchmark's and the served stream's."""
    r = random.Random(c["study"])
    out = []
    for k in range(c["solves"]):
        n = _size(r, c["low"], c["high"])
        adaptive = k % 4 == 3
        d = _steps("", (n, n, n), max(1, c["steps"] // (8 if adaptive else 1)), bcs=r.choice([1, 2]),
                   order=r.choice([2, 4]), storage="c128" if k % 5 == 4 else "c64")
        if adaptive:
            d.update(scheme="rk45", bcs=2, om=0.05, mu=6.0, gamma=0.05, dx=0.25, ic="trap")
        elif d["bcs"] == 2:
            d.update(ic="ring")
        out.append(d)
    return out


def _host(psi, storage):
    """psi in page-locked host memory, as a program that submits many solves keeps its states."""
    a = L.pinned_empty(tuple(psi.shape), np.complex64 if storage == "c64" else np.complex128)
    a[...] = psi.cpu().numpy()
    return a


def prepare(case, seed):
    dev = torch.device("cuda")
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "batch":
        s["solves"] = []
        for k, d in enumerate(_study(case)):
            psi = _host(_state(d, seed * 1000 + k, dev), d["storage"])
            s["solves"].append((_rp(d), psi, d["steps"], L.pinned_empty(psi.shape, psi.dtype)))
        s["pool"] = Pool(sum(Pool.solve_bytes(p) for p, _, _, _ in s["solves"]) + (64 << 20))
    elif kind == "norm":
        dt, s["code"] = _dtypes(case["storage"])
        g = torch.Generator(device=dev).manual_seed(seed)
        shape = (case["nz"], case["ny"], case["nx"])
        s["psi"] = torch.complex(*(torch.randn(shape, generator=g, device=dev, dtype=torch.float64)
                                   for _ in range(2))).to(dt)
        s["norm"] = torch.zeros(1, dtype=torch.float64, device=dev)
        s["lib"] = L.load()
    elif kind == "initial":
        p = _initial_params(case)
        dt, s["code"] = _dtypes(case["storage"])
        s["spec"] = _initial_spec(case, seed)
        s["solver"] = Solver(p)
        s["out"] = torch.empty((p.nz, p.ny, p.nx), dtype=dt, device=dev)
    else:
        p = _rp(case)
        dt, s["code"] = _dtypes(case["storage"])
        s["psi"] = _state(case, seed, dev).to(dt)
        s["solver"] = Solver(p)
        s["out"] = torch.empty_like(s["psi"])
        if kind == "save":
            torch.cuda.synchronize()
            _put(s["solver"], s["psi"], s["code"])
    torch.cuda.synchronize()
    return s


def _put(solver, psi, code):
    rc = solver.lib.gpe_set_state_device(solver.h, C.c_void_p(psi.data_ptr()), code)
    if rc:
        raise L.GpeError(rc, "gpe_set_state_device")


def _get(solver, out, code):
    rc = solver.lib.gpe_get_state_device(solver.h, C.c_void_p(out.data_ptr()), code)
    if rc:
        raise L.GpeError(rc, "gpe_get_state_device")
    return out


def _initial_line(case, seed):
    r = random.Random(seed)
    h = 0.5 * case["dx"] * (min(case["nx"], case["ny"], case["nz"]) - 1)
    return h * r.uniform(-0.2, 0.2), h * r.uniform(-0.2, 0.2), h * r.uniform(0.3, 0.5)


def _initial_params(case):
    h = [0.5 * case["dx"] * (case[a] - 1) for a in ("nx", "ny", "nz")]
    return RunParams(nx=case["nx"], ny=case["ny"], nz=case["nz"], xr=h[0], yr=h[1], zr=h[2], scheme="rk4", bcs=case["bcs"],
                     order=4, g=1.0, mu=case["mu"], omx=case["om"], omy=case["om"], omz=case["om"],
                     storage=case["storage"])


def _initial_spec(case, seed):
    x0, y0, r0 = _initial_line(case, seed)
    return ic.device_spec(*case["factors"].split(","), ring=dict(plane="xy", x0=x0, y0=y0, r0=r0),
                          line=dict(x0=x0, y0=y0, dir="z"))


# ---------------------------------------------------------------------------
# one pass


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "batch":
        pool = s["pool"]
        for k, (p, psi, steps, out) in enumerate(s["solves"]):
            if not pool.submit(p, psi, steps, k, out=out):
                raise RuntimeError("the pool's budget holds every solve of the study")
        res = {r.tag: r for r in pool.run_all()}
        return {"psi": [res[k].psi for k in range(len(res))], "norm": [res[k].norm for k in range(len(res))]}
    if kind == "norm":
        d = case["dx"]
        st = torch.cuda.current_stream().cuda_stream
        rc = s["lib"].gpe_norm_noalloc(C.c_void_p(s["psi"].data_ptr()), s["code"], case["nx"], case["ny"], case["nz"],
                                       d, d, d, C.c_void_p(s["norm"].data_ptr()), C.c_void_p(st))
        if rc:
            raise L.GpeError(rc, "gpe_norm_noalloc")
        return {"norm": s["norm"]}
    sv = s["solver"]
    if kind == "initial":
        sv.set_ic(s["spec"])
        return {"psi": _get(sv, s["out"], s["code"])}
    if kind == "save":
        d = sv.condensed(spectrum=True)
        return {"norm": sv.get_norm(), "energy": sv.energy(), **d}
    _put(sv, s["psi"], s["code"])
    sv.t, sv.im_t, sv.p = 0.0, 0.0, 0
    if kind == "relax":
        sv.dt = complex(0.0, -case["tau"])
        norms = []
        for _ in range(case["steps"]):
            norms.append(sv.solver(1, want_norm=True).norm)
            sv.renormalise(norms[-1])
        return {"psi": _get(sv, s["out"], s["code"]), "norms": norms}
    sv.dt = complex(case["tau"], 0.0)
    info = sv.solver(case["steps"], want_norm=True)
    return {"psi": _get(sv, s["out"], s["code"]), "norm": info.norm, "t": sv.t}


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _rhs_flops(c):
    """Operations of one right-hand side of one site: two parts (real, imaginary) of three axis differences, their
    scaling and sum, and the equation's terms."""
    f = 2 * (3 * ((7 if c["order"] == 4 else 3) + 1) + 2) + 3
    f += {1: 12, 2: 4, 3: 14, 4: 10}[c["eqn"]]
    if c["om"]:
        f += 6
    if c["gamma"]:
        f += 4
    if c["Urhs"]:
        f += 2 * (7 if c["order"] == 4 else 2) + 4
    if c["diss"]:
        f += 8
    return f


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        for d in _study(case):
            w = work(d)
            b += w["bytes"]
            f += w["flops"]
        return {"bytes": b, "flops": f}
    n = case["nx"] * case["ny"] * case["nz"]
    e = 8 if case["storage"] == "c64" else 16
    if kind == "norm":
        return {"bytes": n * e + 8, "flops": 5 * n}
    if kind == "initial":
        return {"bytes": 2 * n * e, "flops": 40 * n}
    if kind == "save":
        # the state is read once; a transform costs 5 n log2 n, the spectra and the temperature sum a few
        # operations a mode
        return {"bytes": n * e, "flops": int(n * (5 * math.log2(n) + 5 + 12 + _rhs_flops(case)))}
    stages = {"euler": 1, "rk2": 2, "rk4": 4, "rk45": 6}[case["scheme"]]
    comb = {"euler": 4, "rk2": 8, "rk4": 26, "rk45": 130}[case["scheme"]]
    # every step reads the state once and writes it once
    return {"bytes": case["steps"] * 2 * n * e, "flops": case["steps"] * n * (stages * _rhs_flops(case) + comb)}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, by plain torch


class _Exact:
    """The stepper's mathematics on (nz, ny, nx) complex128 tensors."""

    def __init__(self, c, dev):
        self.c, self.dev = c, dev
        self.n = (c["nz"], c["ny"], c["nx"])
        h = [0.5 * c["dx"] * (m - 1) for m in self.n]
        self.d = [(a + a) / (m - 1) for a, m in zip(h, self.n)]  # dz, dy, dx
        x, y, z = _axes(c, dev)
        self.v = 0.5 * ((c["om"] ** 2 * (x * x) + c["om"] ** 2 * (y * y)) + c["om"] ** 2 * (z * z))

        def sponge(q):
            a = q.reshape(-1)[-3]
            return 1.0 + torch.tanh(q - a) * torch.tanh(q + a)

        self.diss = c["diss"] * ((sponge(x) + sponge(y)) + sponge(z)) if c["diss"] and c["eqn"] in (1, 3) else 0.0
        self.ball = 0.5 * (1.0 + torch.tanh((torch.sqrt((x * x + y * y) + z * z) - 10.0) - 2.0))
        self.idx = {}
        for ax in range(3):
            m = self.n[ax]
            q = torch.arange(m, device=dev)
            for s in (-2, -1, 1, 2):
                t = q + s
                if c["bcs"] == 1:
                    t = t % m
                else:
                    t = torch.where(t < 0, -t, t)
                    t = torch.where(t > m - 1, 2 * (m - 1) - t, t)
                self.idx[ax, s] = t

    def at(self, p, ax, s):
        return torch.index_select(p, ax, self.idx[ax, s])

    def lap(self, p):
        out = torch.zeros_like(p)
        for ax in range(3):
            d2 = self.d[ax] ** 2
            if self.c["order"] == 2:
                out += (self.at(p, ax, 1) - 2.0 * p + self.at(p, ax, -1)) / d2
            else:
                out += (-self.at(p, ax, 2) + 16.0 * self.at(p, ax, 1) - 30.0 * p + 16.0 * self.at(p, ax, -1)
                        - self.at(p, ax, -2)) / (12.0 * d2)
        return out

    def ddx(self, p):
        d = self.d[2]
        if self.c["order"] == 2:
            return (self.at(p, 2, 1) - self.at(p, 2, -1)) / (2.0 * d)
        return (-self.at(p, 2, 2) + 8.0 * self.at(p, 2, 1) - 8.0 * self.at(p, 2, -1) + self.at(p, 2, -2)) / (12.0 * d)

    @staticmethod
    def n2(p):
        return p.real ** 2 + p.imag ** 2

    def rhs(self, p):
        c = self.c
        if c["eqn"] == 4:
            return -(1j + c["gamma"]) * (-0.5 * self.lap(p) + self.v * p + self.n2(p) * p - c["mu"] * p)
        if c["eqn"] == 2:
            r = 1j * (self.lap(p) - self.n2(p) * p)
        else:
            r = 0.5 * (1j + self.diss) * (self.lap(p) + (1.0 - self.n2(p)) * p)
        if c["Urhs"]:
            r = r + c["Urhs"] * self.ddx(p)
        return r * self.ball if c["eqn"] == 3 else r

    def step(self, p, h):
        sc = self.c["scheme"]
        if sc == "euler":
            return p + h * self.rhs(p)
        if sc == "rk2":
            return p + h * self.rhs(p + 0.5 * h * self.rhs(p))
        k = self.rhs(p)
        acc = k
        k = self.rhs(p + 0.5 * h * k)
        acc = acc + 2.0 * k
        k = self.rhs(p + 0.5 * h * k)
        acc = acc + 2.0 * k
        return p + (h / 6.0) * (acc + self.rhs(p + h * k))

    B = ((0.2,), (0.075, 0.225), (0.3, -0.9, 1.2), (-11.0 / 54.0, 2.5, -70.0 / 27.0, 35.0 / 27.0),
         (1631.0 / 55296.0, 175.0 / 512.0, 575.0 / 13824.0, 44275.0 / 110592.0, 253.0 / 4096.0))
    CO = (37.0 / 378.0, 0.0, 250.0 / 621.0, 125.0 / 594.0, 0.0, 512.0 / 1771.0)
    CE = (2825.0 / 27648.0, 0.0, 18575.0 / 48384.0, 13525.0 / 55296.0, 277.0 / 14336.0, 0.25)

    def adaptive(self, p, h):
        """One accepted Cash-Karp step under the reference's step control: (psi, the step taken, the next)."""
        entry = h
        while True:
            k = [h * self.rhs(p)]
            first = k[0] / h
            for row in self.B:
                q = p.clone()
                for b, km in zip(row, k):
                    q += b * km
                k.append(h * self.rhs(q))
            new, err = p.clone(), torch.zeros_like(p)
            for a, b, km in zip(self.CO, self.CE, k):
                new += a * km
                err += (a - b) * km
            scale = torch.sqrt((torch.abs(p) + entry * torch.abs(first) + 1e-30) ** 2)
            worst = float((torch.abs(err) / scale).max()) / 1e-6
            if worst <= 1.0:
                break
            h = max(0.9 * h * worst ** -0.25, 0.1 * h)
        errcon = (5.0 / 0.9) ** (1.0 / -0.2)
        return new, h, 0.9 * h * worst ** -0.2 if worst > errcon else 5.0 * h

    def norm(self, p):
        s = self.n2(p)
        for ax, m in enumerate(self.n):
            w = torch.ones(m, dtype=torch.float64, device=self.dev)
            for q, v in ((0, 3.0 / 8.0), (1, 7.0 / 6.0), (2, 23.0 / 24.0)):
                w[q] = w[m - 1 - q] = v
            s = s * w.reshape([-1 if a == ax else 1 for a in range(3)])
        return float(s.sum()) * self.d[2] * self.d[1] * self.d[0]

    def energy(self, p):
        e = (-(self.lap(p)) * p.conj()).real + 0.5 * self.n2(p) ** 2
        return float(e.sum()) * self.d[2] * self.d[1] * self.d[0]

    def condensed(self, p):
        """The mass.dat record and the spectra, in the reference's definitions."""
        c = self.c
        nz, ny, nx = self.n
        V = float(nx * ny * nz)
        dz, dy, dx = self.d
        a = torch.fft.fftn(p) / math.sqrt(V)
        v = self.n2(a)
        n0 = float(v[0, 0, 0])
        M = float(self.n2(p).sum()) * dx * dy * dz
        rho0 = n0 / V

        def symbol(m, d):
            k = -PI + torch.arange(m, dtype=torch.float64, device=self.dev) * (2.0 * PI / (nx - 1))
            return ((-2.0 * torch.cos(2.0 * k * d) + 32.0 * torch.cos(k * d)) - 30.0) / (d * d)

        q = -(1.0 / 12.0) * ((symbol(nx, dx)[None, None, :] + symbol(ny, dy)[None, :, None])
                             + symbol(nz, dz)[:, None, None])
        q = q[q != 0.0]
        tot = float(((q + rho0) / (q * q + 2.0 * rho0 * q)).sum())

        def dist2(m):
            i = torch.arange(m, device=self.dev)
            return torch.where(i <= (m - 1) // 2 + 1, i * i, (m - i) ** 2)

        k2 = dist2(nx)[None, None, :] + dist2(ny)[None, :, None] + dist2(nz)[:, None, None]
        # the sums by squared distance first: both spectra depend on it alone
        top = int(k2.max()) + 1
        by = torch.zeros(top, dtype=torch.float64, device=self.dev).index_add_(0, k2.reshape(-1), v.reshape(-1))
        count = torch.bincount(k2.reshape(-1), minlength=top)
        by, count = by.cpu().numpy(), count.cpu().numpy()
        rk = np.sqrt(np.arange(top, dtype=np.float64))
        F = np.array([by[1:][rk[1:] <= kk].sum() for kk in range(1, nx // 2 + 1)])
        al = np.full(top, np.inf)
        al[1:] = np.abs(np.log(0.5 * rk[1:] / PI) / np.log(2.0))
        eta, nharm = np.zeros(7), np.zeros(7, dtype=np.int32)
        for m in range(7):
            sel = (al >= m) & (al < m + 1)
            nharm[m] = count[sel].sum()
            eta[m] = by[sel].sum() / nharm[m] if nharm[m] else 0.0
        temp = (M - n0) / tot
        vol8 = 8.0 * (0.5 * c["dx"]) ** 3 * (nx - 1) * (ny - 1) * (nz - 1)
        return dict(M=M, n0=n0, rho0=rho0, tot=tot, temp=temp, temp2=((M / vol8) - n0 / V) / tot,
                    H=(M ** 2 + (M - n0) ** 2) / (2.0 * V) + temp * (V - 1.0), mass_density=M / vol8, eta=eta,
                    nharm=nharm, F=F)


def _exact_initial(case, seed, dev):
    x, y, z = _axes(case, dev)
    x0, y0, r0 = _initial_line(case, seed)
    psi = torch.ones((case["nz"], case["ny"], case["nx"]), dtype=torch.complex128, device=dev)
    for f in case["factors"].split(","):
        if f == "fermi":
            v = 0.5 * (case["om"] ** 2 * (x * x + y * y + z * z))
            psi = psi * torch.sqrt(torch.clamp(case["mu"] - v, min=0.0))
        elif f == "ring":
            s = torch.sqrt((x - x0) ** 2 + (y - y0) ** 2)
            for b, sign in ((s + r0, 1.0), (s - r0, -1.0)):
                q = _core(torch.sqrt(z * z + b * b))
                psi = psi * torch.complex(q * z, sign * q * b)
        else:
            a, b = x - x0, y - y0
            r, th = torch.sqrt(a * a + b * b), torch.atan2(b, a)
            m = r * _core(r) if f == "line_pade" else 1.0 - torch.exp(-0.7 * r ** 1.15)
            psi = psi * torch.complex(m * torch.cos(th), m * torch.sin(th))
    return psi


def _exact_steps(c, psi, dev):
    """(psi, norm, t) after the case's steps from psi."""
    e = _Exact(c, dev)
    p = psi.to(_dtypes(c["storage"])[0]).to(torch.complex128)
    t = 0.0
    if c["scheme"] == "rk45":
        h = c["tau"]
        for _ in range(c["steps"]):
            p, took, h = e.adaptive(p, h)
            t += took
    else:
        for _ in range(c["steps"]):
            p = e.step(p, c["tau"])
            t += c["tau"]
    return p, e.norm(p), t


def exact(case, seed):
    dev = _device()
    kind = case["kind"]
    if kind == "batch":
        out = [_exact_steps(d, _state(d, seed * 1000 + k, dev), dev) for k, d in enumerate(_study(case))]
        return {"psi": [p for p, _, _ in out], "norm": [m for _, m, _ in out]}
    if kind == "norm":
        s = prepare(case, seed)
        e = _Exact(dict(_steps("", (case["nx"], case["ny"], case["nz"]), 1, dx=case["dx"])), s["psi"].device)
        return {"norm": torch.tensor([e.norm(s["psi"].to(torch.complex128))], dtype=torch.float64)}
    if kind == "initial":
        return {"psi": _exact_initial(case, seed, dev)}
    psi = _state(case, seed, dev)
    if kind == "save":
        e = _Exact(case, dev)
        p = psi.to(_dtypes(case["storage"])[0]).to(torch.complex128)
        return {"norm": e.norm(p), "energy": e.energy(p), **e.condensed(p)}
    if kind == "relax":
        e = _Exact(case, dev)
        p = psi.to(_dtypes(case["storage"])[0]).to(torch.complex128)
        norms = []
        for _ in range(case["steps"]):
            p = e.step(p, -1j * case["tau"])
            norms.append(e.norm(p))
            p = p * (math.sqrt(_norm_goal(case)) / math.sqrt(norms[-1]))
        return {"psi": p, "norms": norms}
    p, norm, t = _exact_steps(case, psi, dev)
    return {"psi": p, "norm": norm, "t": t}
