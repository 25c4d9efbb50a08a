"""Performance cases of the time step and the learned closure.

`listed()` names the cases, `draw()` gives further ones of the same ranges,
`prepare()` sets a case up as a user's program would, `run()` is one timed pass
through the public entry points, `work()` counts what the pass cannot do
without, and `exact()` computes the pass's results in 64 bits with plain torch.

Four kinds of pass:

steps      the state stays on the device: `steps` time steps (`Solver.run`),
           the logged quantities where `log` is set, then every field pulled
           once, as a run that logs and saves at intervals does;
integrate  the reference's own entry point on host arrays: `steps` calls, each
           copying the fields in and out;
rollout    the coarse run with the network's forcing (`closure.run_coarse`);
forward, train   the network by itself: one inference pass, or one update from
           `batch` samples.
"""
from __future__ import annotations

import ctypes
import dataclasses
import math
import tempfile

import numpy as np
import torch

from simpletcsolver_b200 import abi, closure, ic
from simpletcsolver_b200.solver import Solver

FIELDS = ("ux", "uy", "uz", "p", "t")
IN_SCALE = (0.05, 1.0, 0.05)     # network input scales, those of bench.py's closure arm
FORCING = (0.05, 0.05, 0.05)     # scale of the network's output as a forcing
RK_A, RK_B = (32 / 60, 25 / 60, 45 / 60), (0.0, -17 / 60, -25 / 60)


def _steps(nx, ny, nz, Re, steps, curved=True, implicit="x", storage=8, log=False, kind="steps", **more):
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, Re=Re, steps=steps, curved=curved, implicit=implicit, storage=storage,
                log=log, **more)


def _net(kind, nx, ny, nz, batch=1, **more):
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, batch=batch, **more)


def listed():
    return [
        # the reference's "typical" example, run for hundreds of time units with logs in between: the smallest grid
        # in earnest, all launches and latency
        _steps(64, 8, 32, 80.0, 32, log=True, lx=1.0, ly=math.pi / 8, lz=2.0, name="typical_64x8x32"),
        # the CPU-runnable Taylor-Couette workload: a few waves of blocks per kernel
        _steps(64, 128, 64, 3400.0, 32, name="small_64x128x64"),
        # an ordinary production grid, advanced between two logs
        _steps(128, 256, 256, 1.0e4, 16, log=True, name="medium_128x256x256"),
        # the headline Taylor-Couette grid, bench.py's workload
        _steps(256, 1024, 512, 1.0e4, 16, name="large_256x1024x512"),
        # FP32 storage, the option for larger grids and shorter runs
        _steps(128, 512, 256, 1.0e4, 32, storage=4, name="fp32_128x512x256"),
        # the planar channel with every direction implicit, bench.py's second workload
        _steps(192, 512, 256, 2000.0, 16, curved=False, implicit="xyz", name="planar_192x512x256"),
        # lengths that are not powers of two, as FFTW users pick them
        _steps(96, 180, 120, 3400.0, 16, name="ragged_96x180x120"),
        # radial lines longer than 256 points
        _steps(384, 256, 128, 1.0e4, 16, name="radial_384x256x128"),
        # a C host that calls integrate() on its own arrays every step
        _steps(128, 256, 128, 1.0e4, 4, kind="integrate", name="integrate_128x256x128"),
        # the 4x-coarsened run with the learned closure
        _steps(64, 256, 128, 1.0e4, 16, kind="rollout", name="rollout_64x256x128"),
        # the network alone on that grid: inference and one training update
        _net("forward", 64, 256, 128, name="forward_64x256x128"),
        _net("train", 64, 256, 128, batch=4, name="train_64x256x128"),
    ]


def draw(rng):
    def size(lo, hi, multiple):
        """Log-uniform in [lo, hi]: half of the draws a power of two, the others any multiple."""
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        if rng.random() < 0.5:
            return max(lo, min(hi, 2 ** round(math.log2(v))))
        return max(lo, min(hi, multiple * round(v / multiple)))

    kind = rng.choices(("steps", "integrate", "rollout", "forward", "train"), (70, 8, 6, 8, 8))[0]
    if kind in ("rollout", "forward", "train"):
        nx, ny, nz = 8 * rng.randint(1, 8), 16 * rng.randint(1, 16), 4 * rng.randint(2, 32)
        if kind == "rollout":
            return _steps(nx, ny, nz, 1.0e4, rng.randint(2, 16), kind=kind)
        return _net(kind, nx, ny, nz, batch=rng.randint(1, 4) if kind == "train" else 1)
    while True:
        nx, ny, nz = size(12, 512, 1), size(8, 1024, 2), size(8, 512, 4)
        cells = nx * ny * nz
        two = all(n & (n - 1) == 0 for n in (ny, nz))
        if cells <= (4_000_000 if kind == "integrate" else 40_000_000 if two else 16_000_000):
            break
    steps = 4 if kind == "integrate" else max(2, min(32, int((1.5e8 if two else 5e7) / cells)))
    curved = rng.random() < 0.75
    implicit = "x" if curved else rng.choice(("xyz", "xyz", "x"))
    if rng.random() < 0.1:
        implicit = "none"
    storage = 4 if kind == "steps" and rng.random() < 0.25 else 8
    return _steps(nx, ny, nz, rng.choice((2000.0, 3400.0, 1.0e4)), steps, curved=curved, implicit=implicit,
                  storage=storage, log=rng.random() < 0.3, kind=kind)


# ---------------------------------------------------------------- inputs
def _flow(case):
    make = ic.taylor_couette if case["curved"] else ic.plane_couette
    geometry = {k: case[k] for k in ("lx", "ly", "lz") if k in case}
    implicit = tuple(d in case["implicit"] for d in "xyz") if case["implicit"] != "none" else (False,) * 3
    return dataclasses.replace(make(case["nx"], case["ny"], case["nz"], case["Re"]), implicit=implicit, **geometry)


def _initial(case, seed):
    """Laminar profile plus noise on the device, [nz, ny, row] without halos (p = 0); values that single precision
    holds when the state is stored in it."""
    flow = _flow(case)
    nx, ny, nz = flow.nx, flow.ny, flow.nz
    xf, xc = (torch.from_numpy(a).cuda() for a in ic.radial_grid(flow))
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def noise(row, amplitude):
        u = torch.rand(nz, ny, row, generator=gen, device="cuda", dtype=torch.float64)
        return u.sub_(0.5).mul_(2 * amplitude)

    ri, ro = float(xf[0]), float(xf[-1])
    if flow.is_curved:
        a = (flow.uy_xp * ro - flow.uy_xm * ri) / (ro * ro - ri * ri)
        uy = a * xc + (flow.uy_xm - a * ri) * ri / xc
    else:
        uy = flow.uy_xm + (flow.uy_xp - flow.uy_xm) * (xc - ri) / flow.lx
    t = flow.t_xm + (flow.t_xp - flow.t_xm) * (xc - ri) / flow.lx
    f = {"ux": noise(nx + 1, flow.noise_u), "uy": noise(nx + 2, flow.noise_u).add_(uy),
         "uz": noise(nx + 2, flow.noise_u), "p": torch.zeros(nz, ny, nx + 2, dtype=torch.float64, device="cuda"),
         "t": noise(nx + 2, flow.noise_t).add_(t)}
    if case["storage"] == 4:
        f = {n: v.float().double() for n, v in f.items()}
    f["ux"][..., 0] = f["ux"][..., -1] = 0.0
    for n, lo, hi in (("uy", flow.uy_xm, flow.uy_xp), ("uz", 0.0, 0.0), ("t", flow.t_xm, flow.t_xp)):
        f[n][..., 0], f[n][..., -1] = lo, hi
    return f


def _parameters(seed):
    """Weights and biases of the network's layers, [27][cout][cin] and [cout], FP32 on the host."""
    rng = np.random.default_rng(seed)
    out = []
    for cin, _, cout, _ in closure.LAYERS:
        std = math.sqrt(2.0 / (27 * cin))
        out.append((rng.normal(0.0, std, (27, cout, cin)).astype(np.float32),
                    rng.normal(0.0, 0.02, cout).astype(np.float32)))
    return out


def _samples(case, seed):
    """Network inputs (BF16 [batch][cell][16], channels as the closure fills them) and targets (FP32 [batch][cell][3])."""
    nx, ny, nz, batch = case["nx"], case["ny"], case["nz"], case["batch"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.zeros(batch, nz, ny, nx, closure.NIN, device="cuda")
    x[..., :3] = torch.randn(batch, nz, ny, nx, 3, generator=gen, device="cuda")
    x[..., 3] = 2.0 * (torch.arange(nx, device="cuda") + 0.5) / nx - 1.0
    y = torch.randn(batch, nz, ny, nx, closure.NOUT, generator=gen, device="cuda")
    return x.bfloat16(), y


class _Flow:
    """A solver and its host arrays, both given back with the object (the arrays are the caller's to free)."""

    def __init__(self, case, seed):
        flow, kind = _flow(case), case["kind"]
        with tempfile.TemporaryDirectory() as d:
            s = self.solver = Solver.from_case(flow, d, storage=case["storage"])
        self.free = ctypes.CDLL(None).free
        self.free.argtypes = [ctypes.c_void_p]
        members = [getattr(s.fluid, name) for name, _ in abi.FluidT._fields_]
        self.arrays = [m for m in members if isinstance(m, abi.ArrayT)]
        self.arrays += [a for m in members if isinstance(m, abi.ArrayT * 3) for a in m]
        s.set_coherence(abi.PIN_HOST | (0 if kind == "integrate" else abi.NO_COHERENCE))
        for n, v in _initial(case, seed).items():
            torch.from_numpy(s.field(n))[1:-1, 1:-1].copy_(v)
        s.push()
        if kind == "integrate":
            s.pull()     # the host arrays with their walls and periodic images, which integrate() reads

    def field(self, name):
        """The host array, which keeps this object alive."""
        s = self.solver
        row = s.nx + 1 if name == "ux" else s.nx + 2
        buf = (ctypes.c_double * (row * (s.ny + 2) * (s.nz + 2))).from_address(getattr(s.fluid, name).data)
        buf.owner = self
        return np.frombuffer(buf, dtype=np.float64).reshape(s.nz + 2, s.ny + 2, row)

    def fields(self):
        return {n: self.field(n) for n in FIELDS}

    def __del__(self):
        if getattr(self, "solver", None) is None:
            return
        self.solver.release()
        for a in self.arrays:
            self.free(a.data)


def prepare(case, seed):
    state = dict(case)
    if case["kind"] in ("forward", "train", "rollout"):
        params = _parameters(seed)
        net = state["net"] = closure.ClosureNet(abi.load(), (case["nx"], case["ny"], case["nz"]))
        net.load_state(np.concatenate([v.ravel() for layer in params for v in layer]))
    if case["kind"] in ("forward", "train"):
        x, y = _samples(case, seed)
        state["x"], state["y"] = x.flatten(1), y.flatten(1)
        # a training that is under way: moments of earlier updates
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        net.m.copy_(1e-3 * torch.randn(net.m.shape, generator=gen, device="cuda"))
        net.v.fill_(1e-6)
        net.adam_steps = 1000
        torch.cuda.synchronize()
    else:
        state["flow"] = _Flow(case, seed)
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "forward":
        return {"out": state["net"].forward(state["x"][0], keep=False)}
    if kind == "train":
        net = state["net"]
        net.loss.zero_()
        for q in range(state["batch"]):
            net.forward(state["x"][q])
            net.backward(state["y"][q], x=state["x"][q], accumulate=q > 0)
        net.adam(1e-3)
        return {"loss": net.loss, "grads": net.grads, "params": net.params, "m": net.m, "v": net.v}
    flow = state["flow"]
    s = flow.solver
    if kind == "integrate":
        dts = np.array([s.integrate() for _ in range(state["steps"])])
        return {"dt": dts, **flow.fields()}
    if kind == "rollout":
        times, _ = closure.run_coarse(s, math.inf, state["net"], IN_SCALE, FORCING, max_steps=state["steps"])
        out = {"dt": np.diff(times)}
    else:
        out = {"dt": s.run(state["steps"])}
        if state["log"]:
            out["log"] = np.array(list(s.log_quantities().values()))
    s.pull(abi.UX | abi.UY | abi.UZ | abi.P | abi.T)
    fields = flow.fields()
    if kind == "rollout" or state["storage"] == 4:
        # a state that is worth single precision goes on to its users, on the device, in single precision
        fields = {n: torch.from_numpy(v).cuda().float() for n, v in fields.items()}
    return {**out, **fields}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes and operations of one pass. A step's stages each read their inputs and write their outputs once (the
    global transforms keep them apart): the predict reads five fields and writes four fields and the four source
    terms (the later two substeps read the former sources too), divergence and y transform, z transform, radial solves,
    z transform, y transform, correction; implicit y and z add two passes over the increments each and the update."""
    cells = case["nx"] * case["ny"] * case["nz"]
    layers = [2 * 27 * cin * cout for cin, _, cout, _ in closure.LAYERS]
    if case["kind"] == "forward":
        return {"bytes": cells * (2 * closure.NIN + 4 * closure.NOUT), "flops": cells * sum(layers)}
    if case["kind"] == "train":
        one = cells * (3 * sum(layers) - layers[0])
        return {"bytes": case["batch"] * cells * (2 * closure.NIN + 4 * closure.NOUT), "flops": case["batch"] * one}
    if case["storage"] == 4:
        step = 56 + 72 + 72 + 3 * (16 + 8 + 8 + 8 + 12 + 48)
    else:
        step = 104 + 136 + 136 + 3 * (32 + 16 + 16 + 16 + 16 + 72)
    if "y" in case["implicit"]:
        step += 3 * (2 * 64 + 64)
    pulled = 8 * len(FIELDS)
    fft = 5.0 * (math.log2(case["ny"]) + 2 * math.log2(case["nz"]))
    flops = 3 * (330 + fft)
    if case["kind"] == "rollout":
        step += 3 * 24 + 2 * closure.NIN + 8 * closure.NOUT
        flops += sum(layers)
    if case["kind"] == "integrate":
        return {"bytes": cells * case["steps"] * (step + 2 * pulled + 8), "flops": cells * case["steps"] * flops}
    return {"bytes": cells * (case["steps"] * step + pulled), "flops": cells * case["steps"] * flops}


# ---------------------------------------------------------------- the same in 64 bits, plain torch
def _network(x, params):
    """x [cell..., 16] as [nz, ny, nx, 16] -> [nz, ny, nx, 3], FP64."""
    h = x[..., :4].double()
    for li, (w, b) in enumerate(params):
        co, ci = w.shape[1:]
        h = h.permute(3, 0, 1, 2)[None]
        h = torch.nn.functional.pad(h, (0, 0, 1, 1, 1, 1), mode="circular")
        h = torch.nn.functional.pad(h, (1, 1))
        h = torch.nn.functional.conv3d(h, w.reshape(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2), b)[0].permute(1, 2, 3, 0)
        if li < len(params) - 1:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    return h


class _Exact:
    """One flow advanced in FP64 with whole-array operations: ux [nz, ny, nx+1] at the faces, the others
    [nz, ny, nx+2] with their wall columns, periodic in y and z."""

    def __init__(self, case, seed):
        self.case, self.flow = case, _flow(case)
        flow = self.flow
        self.n = nx, ny, nz = flow.nx, flow.ny, flow.nz
        xf, xc = (torch.from_numpy(a).cuda() for a in ic.radial_grid(flow))
        hf, hc = xc[1:] - xc[:-1], torch.empty_like(xc)
        hc[1:-1] = xf[1:] - xf[:-1]
        hc[0], hc[-1] = 0.5 * (xf[1] - xf[0]), 0.5 * (xf[-1] - xf[-2])
        rf, rc = (xf, xc) if flow.is_curved else (torch.ones_like(xf), torch.ones_like(xc))
        self.hf, self.hc, self.hz = hf, hc, flow.lz / nz
        self.yf, self.yc = rf * flow.ly / ny, rc * flow.ly / ny
        self.Jf, self.Jc = hf * self.yf * self.hz, hc * self.yc * self.hz
        self.a, self.b = self.Jf / hf, self.Jc / hc
        self.nu, self.kappa = 1.0 / flow.Re, 1.0 / flow.Re / flow.Pr
        # radial Laplacians: lower and upper coefficients at the inner faces and at the centres
        self.lx = {"ux": (self.b[1:-2] / hc[1:-2] / self.Jf[1:-1], self.b[2:-1] / hc[2:-1] / self.Jf[1:-1])}
        for v in ("uy", "uz", "t"):
            self.lx[v] = (self.a[:-1] / hf[:-1] / self.Jc[1:-1], self.a[1:] / hf[1:] / self.Jc[1:-1])
        self.f = _initial(case, seed)
        self.old = None

    @staticmethod
    def at(q, j=0, k=0):
        return torch.roll(q, (-k, -j), (0, 1)) if j or k else q

    def next_dt(self):
        flow, f, small = self.flow, self.f, 1e-8
        dt = min(1.0, float((self.hf[1:-1] / (f["ux"][..., 1:-1].abs() + small)).min()),
                 float((self.yc[1:-1] / (f["uy"][..., 1:-1].abs() + small)).min()),
                 float((self.hz / (f["uz"][..., 1:-1].abs() + small)).min())) * flow.coef_dt_adv
        for h, implicit in zip((float(self.hc.min()), float(self.yc[1]), self.hz), flow.implicit):
            if not implicit:
                dt = min(dt, flow.coef_dt_dif / max(self.nu, self.kappa) / 6.0 * h * h)
        return dt

    def sides(self):
        """Explicit and implicit right-hand sides of every variable at its unknowns."""
        at, f, nu = self.at, self.f, self.nu
        ux, uy, uz, p, t = (f[n] for n in FIELDS)
        Jf, Jc, a, hz = self.Jf[1:-1], self.Jc[1:-1], self.a, self.hz
        U, V, W = a * ux, (self.Jc / self.yc * uy)[..., 1:-1], (self.Jc / hz * uz)[..., 1:-1]
        da, db = a[1:] - a[:-1], self.b[1:] - self.b[:-1]
        uxc, uyi, uzi = ux[..., :-1] + ux[..., 1:], uy[..., 1:-1], uz[..., 1:-1]
        weight = torch.full_like(uy[0, 0], 0.5)
        weight[0] = weight[-1] = 0.0
        wuy = weight * uy
        lyx1 = -db / self.Jf * (wuy[..., :-1] + wuy[..., 1:])
        lxy = (uy[..., 1:] - uy[..., :-1]) / self.hf
        lxz = (uz[..., 1:] - uz[..., :-1]) / self.hf
        lyx = (ux - at(ux, -1)) / self.yf + lyx1
        lyy1 = 0.5 * da / Jc * uxc
        lyy = (at(uyi, 1) - uyi) / self.yc[1:-1] + lyy1
        lyz = (uzi - at(uzi, -1)) / self.yc[1:-1]
        lzx = (ux - at(ux, 0, -1)) / hz
        lzy = (uyi - at(uyi, 0, -1)) / hz

        def mean_x(q):
            return 0.5 * (q[..., :-1] + q[..., 1:])

        def carried(flux, q, J, lo, hi):
            """-(skew-symmetric advection) of q by the fluxes through two opposite faces."""
            return 0.5 * (flux[0] * (lo - q) - flux[1] * (hi - q)) / J

        e, g = {}, {}
        diffusion = {"ux": (2, 1, 1), "uy": (1, 2, 1), "uz": (1, 1, 2), "t": (1, 1, 1)}
        for v in ("ux", "uy", "uz", "t"):
            full = f[v]
            q, lo, hi = full[..., 1:-1], full[..., :-2], full[..., 2:]
            if v == "ux":
                J, h = Jf, self.yf[1:-1]
                Fx = (mean_x(U)[..., :-1], mean_x(U)[..., 1:])
                Fy, Fz = (mean_x(V), at(mean_x(V), 1)), (mean_x(W), at(mean_x(W), 0, 1))
            else:
                J, h = Jc, self.yc[1:-1]
                if v == "uy":
                    m, Fy = 0.5 * (U + at(U, -1)), (0.5 * (at(V, -1) + V), 0.5 * (V + at(V, 1)))
                    Fz = 0.5 * (W + at(W, -1))
                    Fz = (Fz, at(Fz, 0, 1))
                elif v == "uz":
                    m, Fy = 0.5 * (U + at(U, 0, -1)), 0.5 * (V + at(V, 0, -1))
                    Fy, Fz = (Fy, at(Fy, 1)), (0.5 * (at(W, 0, -1) + W), 0.5 * (W + at(W, 0, 1)))
                else:
                    m, Fy, Fz = U, (V, at(V, 1)), (W, at(W, 0, 1))
                Fx = (m[..., :-1], m[..., 1:])
            e[v] = carried(Fx, q, J, lo, hi) + carried(Fy, q, J, at(q, -1), at(q, 1))
            e[v] += carried(Fz, q, J, at(q, 0, -1), at(q, 0, 1))
            g[v] = torch.zeros_like(q)
            d = self.kappa if v == "t" else nu
            laplacian = (self.lx[v][0] * (lo - q) + self.lx[v][1] * (hi - q),
                         (at(q, -1) - 2 * q + at(q, 1)) / h / h, (at(q, 0, -1) - 2 * q + at(q, 0, 1)) / hz / hz)
            for implicit, c, term in zip(self.flow.implicit, diffusion[v], laplacian):
                (g if implicit else e)[v] += c * d * term
        # curvature and cross diffusion
        uyc = 0.5 * (uyi + at(uyi, 1))
        s = lyx1 + lxy
        e["ux"] += 0.5 / Jf * ((da * uyc * uyc)[..., :-1] + (da * uyc * uyc)[..., 1:])
        e["ux"] += nu * ((at(s, 1) - s)[..., 1:-1] / self.yf[1:-1] + (at(lxz, 0, 1) - lxz)[..., 1:-1] / hz)
        e["ux"] -= nu / Jf * ((da * lyy)[..., :-1] + (da * lyy)[..., 1:])
        e["uy"] -= 0.125 * da / Jc * ((uyi + at(uyi, -1)) * at(uxc, -1) + (uyi + at(uyi, 1)) * uxc)
        e["uy"] += nu / Jc * ((a * lyx)[..., 1:] - (a * lyx)[..., :-1])
        e["uy"] += nu * (2 * (lyy1 - at(lyy1, -1)) / self.yc[1:-1] + (at(lyz, 0, 1) - lyz) / hz)
        r = db * (lyx + lxy)
        e["uy"] += 0.5 * nu / Jc * (r[..., :-1] + r[..., 1:])
        e["uz"] += nu / Jc * ((a * lzx)[..., 1:] - (a * lzx)[..., :-1]) + nu * (at(lzy, 1) - lzy) / self.yc[1:-1]
        pi = p[..., 1:-1]
        g["ux"] -= (pi[..., 1:] - pi[..., :-1]) / self.hf[1:-1]
        g["uy"] -= (pi - at(pi, -1)) / self.yc[1:-1]
        g["uz"] -= (pi - at(pi, 0, -1)) / hz
        return e, g

    def implicit(self, v, delta, pf):
        """(I - pf d2/dx2)(I - pf d2/dy2)(I - pf d2/dz2) inverted on delta, one direction after the other."""
        double = {"ux": 0, "uy": 1, "uz": 2, "t": 1}[v]
        ix, iy, iz = self.flow.implicit
        if ix:
            c = pf * (2 if double == 0 else 1)
            lo, hi = self.lx[v]
            m = torch.diag(1 + c * (lo + hi)) - torch.diag(c * lo[1:], -1) - torch.diag(c * hi[:-1], 1)
            delta = delta @ torch.linalg.inv(m).T
        h = (self.yf if v == "ux" else self.yc)[1:-1]
        for on, dim, n, step in ((iy, 1, self.n[1], h), (iz, 0, self.n[2], self.hz)):
            if on:
                c = pf * (2 if double == (1 if dim else 2) else 1)
                wave = 4 * torch.sin(torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64) * math.pi / n) ** 2
                scale = 1 + c * wave.reshape((-1, 1) if dim else (-1, 1, 1)) / step / step
                delta = torch.fft.irfft(torch.fft.rfft(delta, dim=dim) / scale, n=n, dim=dim)
        return delta

    def potential(self, gdt):
        at, f, a, hz = self.at, self.f, self.a, self.hz
        nx, ny, nz = self.n
        U, V, W = a * f["ux"], (self.Jc / self.yc * f["uy"])[..., 1:-1], (self.Jc / hz * f["uz"])[..., 1:-1]
        div = (U[..., 1:] - U[..., :-1] + at(V, 1) - V + at(W, 0, 1) - W) / self.Jc[1:-1]
        q = torch.fft.fft(torch.fft.rfft(div / gdt, dim=1), dim=0).permute(2, 0, 1).contiguous()
        ey, ez = (4 * torch.sin(torch.arange(m, device="cuda", dtype=torch.float64) * math.pi / n) ** 2
                  for m, n in ((ny // 2 + 1, ny), (nz, nz)))
        lo, hi = self.lx["uy"]
        v = torch.empty(q.shape, dtype=torch.float64, device="cuda")
        for i in range(nx):
            c = -(lo[i] if i else 0 * lo[i]) - (hi[i] if i < nx - 1 else 0 * hi[i])
            c = c - ey[None, :] / self.yc[i + 1] ** 2 - ez[:, None] / hz ** 2
            if i:
                c = c - lo[i] * v[i - 1]
                q[i] -= lo[i] * q[i - 1]
            if i == nx - 1:
                c[0, 0], q[i, 0, 0] = 1.0, 0.0     # the mean's free constant
            v[i] = hi[i] / c
            q[i] /= c
        for i in range(nx - 2, -1, -1):
            q[i] -= v[i] * q[i + 1]
        psi = torch.fft.irfft(torch.fft.ifft(q.permute(1, 2, 0), dim=0), n=ny, dim=1)
        return torch.cat((psi[..., :1], psi, psi[..., -1:]), dim=2)

    def substep(self, rk, dt, forcing=None):
        at, f = self.at, self.f
        e, g = self.sides()
        if forcing is not None:
            e["ux"] += forcing[..., 1:, 0]
            e["uy"] += forcing[..., 1]
            e["uz"] += forcing[..., 2]
        gamma = RK_A[rk] + RK_B[rk]
        for v in e:
            delta = dt * (RK_A[rk] * e[v] + gamma * g[v])
            if rk:
                delta += dt * RK_B[rk] * self.old[v]
            d = self.kappa if v == "t" else self.nu
            f[v] = f[v].clone()
            f[v][..., 1:-1] += self.implicit(v, delta, 0.5 * gamma * dt * d)
        self.old = e
        gdt = gamma * dt
        psi = self.potential(gdt)
        c = psi[..., 1:-1]
        f["ux"][..., 1:-1] -= gdt * (c[..., 1:] - c[..., :-1]) / self.hf[1:-1]
        f["uy"][..., 1:-1] -= gdt * (c - at(c, -1)) / self.yc[1:-1]
        f["uz"][..., 1:-1] -= gdt * (c - at(c, 0, -1)) / self.hz
        lo, hi = self.lx["uy"]
        laplacian = (lo * (psi[..., :-2] - c) + hi * (psi[..., 2:] - c),
                     (at(c, -1) - 2 * c + at(c, 1)) / self.yc[1:-1] ** 2,
                     (at(c, 0, -1) - 2 * c + at(c, 0, 1)) / self.hz ** 2)
        p = f["p"][..., 1:-1] + c
        for implicit, term in zip(self.flow.implicit, laplacian):
            if implicit:
                p = p - gdt * self.nu * term
        f["p"] = torch.cat((p[..., :1], p, p[..., -1:]), dim=2)

    def halos(self):
        nx, ny, nz = self.n
        j, k = ((torch.arange(n + 2, device="cuda") - 1) % n for n in (ny, nz))
        return {n: self.f[n][k][:, j] for n in FIELDS}


def exact(case, seed):
    kind = case["kind"]
    params = [tuple(torch.from_numpy(v).cuda().double() for v in layer) for layer in _parameters(seed)]
    if kind == "forward":
        x, _ = _samples(case, seed)
        return {"out": _network(x[0], params).reshape(-1)}
    if kind == "train":
        x, y = _samples(case, seed)
        flat = [v.requires_grad_() for layer in params for v in layer]
        grads, loss = [torch.zeros_like(v) for v in flat], 0.0
        for q in range(case["batch"]):
            one = ((_network(x[q], params) - y[q]) ** 2).mean()
            loss += one.item()
            for total, part in zip(grads, torch.autograd.grad(one, flat)):
                total += part
        g = torch.cat([v.reshape(-1) for v in grads])
        p = torch.cat([v.detach().reshape(-1) for v in flat])
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        m = 0.9 * (1e-3 * torch.randn(p.shape, generator=gen, device="cuda")).double() + 0.1 * g
        v = 0.999 * torch.full_like(p, 1e-6) + 0.001 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** 1001)) / (torch.sqrt(v / (1 - 0.999 ** 1001)) + 1e-8)
        return {"loss": torch.tensor([loss], dtype=torch.float64), "grads": g, "params": p, "m": m, "v": v}
    if case["nx"] * case["ny"] * case["nz"] * case["steps"] > 1_000_000_000:
        return None     # minutes
    flow = _Exact(case, seed)
    dts = []
    for _ in range(case["steps"]):
        forcing = None
        if kind == "rollout":
            ux, uy, uz = (flow.f[n] for n in ("ux", "uy", "uz"))
            x = torch.zeros(*uy.shape[:2], case["nx"], 4, dtype=torch.float64, device="cuda")
            x[..., 0] = 0.5 * (ux[..., :-1] + ux[..., 1:]) / IN_SCALE[0]
            x[..., 1], x[..., 2] = uy[..., 1:-1] / IN_SCALE[1], uz[..., 1:-1] / IN_SCALE[2]
            x[..., 3] = 2.0 * (torch.arange(case["nx"], device="cuda") + 0.5) / case["nx"] - 1.0
            forcing = _network(x, params) * torch.tensor(FORCING, device="cuda")
        dts.append(flow.next_dt())
        for rk in range(3):
            flow.substep(rk, dts[-1], forcing)
    out = {"dt": torch.tensor(dts, dtype=torch.float64), **flow.halos()}
    if case["kind"] == "steps" and case["log"]:
        out["log"] = None
    return out
