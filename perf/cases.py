"""The work that is timed: what a program that uses this framework has it do, through its public entry
points (nse2d_b200.Solver, Ensemble, Cnn), from the smallest channels to the production grid.

A case is a dict of plain values; `kind` says which calls a pass makes:

  step      nsteps SSPRK(3,3) steps of a channel that is stepped from the host, and its fields
            (precision 64, or 32 for the FP32-bulk variant, whose fields are read at that precision)
  run       the device-side time loop between two outputs, as the executable runs it: nsteps steps by
            Solver.run, then t and one diagnostics row
  ensemble  steps of a batch of uneven channels by one launch
  poisson   the streamfunction solve alone, on the caller's buffers
  closure   steps of a coarse channel whose right-hand side carries the learned subgrid term
  train     one training step of the closure model on a batch of fields, and its gradients
  sample    what an output interval costs: diagnostics row, profile moments, spectra
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "nse2d-channel-gpu_b200"))
import nse2d_b200 as nse  # noqa: E402

F64 = torch.float64
LX = 2.0 * math.pi


# ---- the cases ----

def listed():
    return [
        # the smallest channel that is stepped in earnest (verification and smoke runs): latency and launches
        dict(name="step64_128x129", kind="step", precision=64, Nx=128, Ny=129, beta=2.0, Reb=2000.0, nforce=4, nsteps=10),
        # the small plain-method channel through the executable's time loop, 40 steps between outputs
        dict(name="run64_256x257", kind="run", precision=64, Nx=256, Ny=257, beta=2.0, Reb=5000.0, nforce=8, nsteps=40),
        # the reference's default size class, FP64
        dict(name="step64_1024x513", kind="step", precision=64, Nx=1024, Ny=513, beta=2.0, Reb=1e4, nforce=8, nsteps=4),
        # the DNS that the closure is trained from
        dict(name="step64_2048x1025", kind="step", precision=64, Nx=2048, Ny=1025, beta=1.75, Reb=1e4, nforce=8, nsteps=2),
        # the production size, one step per call (its grid is stretched less than the benchmark's, so that round-off
        # at the first wall spacing stays comparable)
        dict(name="step64_4096x2049", kind="step", precision=64, Nx=4096, Ny=2049, beta=1.2, Reb=2e4, nforce=12, nsteps=1),
        # FP32 bulk: an ensemble-sized channel with a row count that is not 2^k + 1, and the production size
        dict(name="step32_512x301", kind="step", precision=32, Nx=512, Ny=301, beta=2.0, Reb=5000.0, nforce=8, nsteps=8),
        dict(name="step32_4096x2049", kind="step", precision=32, Nx=4096, Ny=2049, beta=2.0, Reb=2e4, nforce=12, nsteps=4),
        # a batch of uneven channels in one launch
        dict(name="ensemble64_12", kind="ensemble", precision=64, members=12, nsteps=5),
        # a program that keeps its own time loop and calls the streamfunction solve (ragged row count)
        dict(name="poisson_1024x777", kind="poisson", Nx=1024, Ny=777, beta=1.5),
        # the coarse solve with the learned closure
        dict(name="closure_256x129", kind="closure", Nx=256, Ny=129, beta=2.0, Reb=1e4, nforce=8, hidden=32, nsteps=5),
        # training of the closure model: batch of 8 coarse fields
        dict(name="train_256x129_b8", kind="train", Nx=256, Ny=129, beta=2.0, hidden=32, batch=8),
        # an output interval of an ordinary run
        dict(name="sample_1024x513", kind="sample", precision=64, Nx=1024, Ny=513, beta=2.0, Reb=1e4, nforce=8),
    ]


def _beta(r, Ny):
    """A stretching whose first wall spacing keeps the wall closure's round-off comparable at this row count."""
    if Ny <= 600:
        return r.choice([0.0, 1.5, 2.0])
    if Ny <= 1100:
        return r.choice([0.0, 1.25, 1.75])
    return r.choice([0.0, 1.0, 1.2])


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step32", "step32", "run", "ensemble", "poisson", "closure", "train", "sample"])
    if kind == "ensemble":
        return dict(kind=kind, precision=rng.choice([64, 64, 32]), members=rng.randint(4, 16), nsteps=rng.randint(3, 6))
    if kind in ("closure", "train"):
        Nx = rng.choice([64, 128, 256])
        c = dict(kind=kind, Nx=Nx, Ny=rng.randint(Nx // 2 - 15, Nx // 2 + 33), beta=2.0, hidden=rng.choice([16, 32, 48, 64]))
        if kind == "closure":
            c.update(Reb=rng.choice([5e3, 1e4]), nforce=rng.choice([4, 8]), nsteps=rng.randint(3, 6))
        else:
            c.update(batch=rng.randint(1, 12))
        return c
    precision = 32 if kind == "step32" else 64
    kind = "step" if kind == "step32" else kind
    Nx = 2 ** rng.randint(6, 12 if kind in ("step", "poisson") else 10)
    Ny = int(math.exp(rng.uniform(math.log(max(33, Nx // 4)), math.log(max(65, Nx // 2 + 1)))))
    c = dict(kind=kind, Nx=Nx, Ny=Ny, beta=_beta(rng, Ny))
    if kind == "poisson":
        return c
    c.update(precision=precision, Reb=round(math.exp(rng.uniform(math.log(2e3), math.log(2e4))), 1), nforce=rng.choice([4, 8, 12]))
    if kind == "step":
        c["nsteps"] = max(1, min(10, int(round(2.0e6 / (Nx * Ny)))))
    elif kind == "run":
        c["nsteps"] = rng.randint(20, 50)
    return c


# ---- inputs ----

def _y(Ny, beta):
    e = -1.0 + 2.0 * np.arange(Ny) / (Ny - 1)
    return np.tanh(beta * e) / np.tanh(beta) if beta > 0 else -1.0 + np.arange(Ny) * (2.0 / (Ny - 1))


def _cfg(case):
    return dict(Nx=case["Nx"], Ny=case["Ny"], Lx=LX, h=1.0, stretch=1 if case["beta"] > 0 else 0, beta=case["beta"], Ub=1.0,
                Reb=case.get("Reb", 1e4), F0=0.05, nforce=case.get("nforce", 8), lin_drag=1e-3, adapt=1, cfl=0.5, dt_max=1e-2,
                dt_init=1e-3, precision=case.get("precision", 64))


def _omega(Nx, Ny, beta, seed, amp=0.05):
    """The 'mix' start: Poiseuille vorticity plus seeded random vorticity over the streamwise modes 1..64; Poiseuille on the walls."""
    rng = np.random.default_rng(seed)
    M = min(64, Nx // 2 - 1)
    A = amp * rng.standard_normal(M) / np.sqrt(M)
    phi = 2 * np.pi * rng.random(M)
    p = rng.integers(1, 9, size=M)
    t = lambda a: torch.tensor(a, dtype=F64, device="cuda")  # noqa: E731
    y = t(_y(Ny, beta))
    x = torch.arange(Nx, dtype=F64, device="cuda") * (LX / Nx)
    k = t(np.arange(1, M + 1) * (2 * np.pi / LX))
    C = t(A)[:, None] * torch.cos(k[:, None] * x[None, :] + t(phi)[:, None])
    S = torch.sin(t(p.astype(float))[:, None] * math.pi * (y[None, :] + 1.0) / 2.0)
    w = (3.0 * y)[:, None] + S.T @ C
    w[0] = 3.0 * y[0]
    w[-1] = 3.0 * y[-1]
    return w.contiguous()


def _members(case, seed):
    """The batch: (Nx, Ny) from {256, 512, 1024} x {129, 257, 513}, Re_b log-uniform in [2e3, 2e4]."""
    r = random.Random(1000 * case["members"] + case["nsteps"])     # the sizes are the case's; the fields are the seed's
    out = []
    for i in range(case["members"]):
        out.append(dict(Nx=r.choice([256, 512, 1024]), Ny=r.choice([129, 257, 513]), beta=2.0, precision=case["precision"],
                        Reb=math.exp(r.uniform(math.log(2e3), math.log(2e4))), nforce=r.choice([4, 8, 12]), seed=100 * seed + i))
    return out


def _net(case, seed, max_batch):
    net = nse.Cnn(case["Nx"], case["Ny"], _y(case["Ny"], case["beta"]), case["hidden"], max_batch)
    net.init_params(seed)
    net.set_scales(*_SCALES)
    return net


_SCALES = ([2.0, 0.75, 0.6, 0.1], 10.0)      # omega, psi, u, v; tau


def _fields(case, seed, samples):
    """Coarse training fields [samples, Ny, Nx]: omega of the 'mix' start, psi, u, v and the subgrid term tau, all smooth random fields of a channel's magnitudes."""
    Nx, Ny = case["Nx"], case["Ny"]
    y = torch.tensor(_y(Ny, case["beta"]), dtype=F64, device="cuda")
    w = torch.stack([_omega(Nx, Ny, case["beta"], 1000 * seed + s, 1.0) for s in range(samples)])
    g = [torch.stack([_omega(Nx, Ny, case["beta"], 1000 * seed + 100 * q + s, 1.0) for s in range(samples)]) - (3.0 * y)[:, None] for q in range(1, 5)]
    psi = (1.5 * (y - y ** 3 / 3.0) + 1.0)[:, None] + 0.1 * g[0]
    u = (1.5 * (1.0 - y ** 2))[:, None] + 0.2 * g[1]
    v = 0.1 * g[2]
    tau = 10.0 * g[3] + 5.0 * (w - (3.0 * y)[:, None])
    tau[:, 0] = 0.0
    tau[:, -1] = 0.0
    return [a.contiguous() for a in (w, psi, u, v, tau)]


class _Device:
    """A field of a solver, as its device pointer; the solver lives as long as a tensor made of it."""

    def __init__(self, s, which):
        self.solver = s
        self.__cuda_array_interface__ = {"shape": (s.Ny, s.Nx), "typestr": "<f8", "data": (s.field_ptr(which), False), "version": 3}


def _view(s, which):
    return torch.as_tensor(_Device(s, which), device="cuda")


def _solver(case, seed):
    s = nse.Solver(**_cfg(case))
    s.set_omega(_omega(case["Nx"], case["Ny"], case["beta"], seed))
    return s


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("step", "run", "sample", "closure"):
        st["solver"] = s = _solver(case, seed)
        if kind == "closure":
            st["net"] = net = _net(case, seed, 1)
            net.set_application(1, 0.25, True)               # the mean-flow mode, which is the one that runs stably
            s.set_closure(net, every_stage=True)
        if case.get("precision", 64) == 64:
            st["out"] = [_view(s, 0), _view(s, 1)]
        else:
            st["wide"] = [torch.empty((s.Ny, s.Nx), dtype=F64, device="cuda") for _ in range(2)]
            st["out"] = [torch.empty((s.Ny, s.Nx), dtype=torch.float32, device="cuda") for _ in range(2)]
    elif kind == "ensemble":
        st["members"] = m = _members(case, seed)
        st["solvers"] = [_solver(c, c["seed"]) for c in m]
        st["ensemble"] = nse.Ensemble(st["solvers"])
        if case["precision"] == 64:
            st["out"] = [[_view(s, 0), _view(s, 1)] for s in st["solvers"]]
        else:
            st["wide"] = [[torch.empty((s.Ny, s.Nx), dtype=F64, device="cuda") for _ in range(2)] for s in st["solvers"]]
            st["out"] = [[torch.empty((s.Ny, s.Nx), dtype=torch.float32, device="cuda") for _ in range(2)] for s in st["solvers"]]
    elif kind == "poisson":
        st["solver"] = nse.Solver(**_cfg(case))
        st["w"] = _omega(case["Nx"], case["Ny"], case["beta"], seed)
        st["psi"] = torch.zeros_like(st["w"])
    elif kind == "train":
        st["net"] = _net(case, seed, case["batch"])
        st["fields"] = _fields(case, seed, case["batch"] + 3)
        st["idx"] = np.random.default_rng(seed).permutation(case["batch"] + 3)[:case["batch"]].astype(np.int32)
    return st


# ---- a pass ----

def _read32(s, wide, out):
    """The fields of an FP32-bulk channel, on the device and at its precision."""
    if s.lib.nse2d_get_fields(s.h, ctypes.c_void_p(wide[0].data_ptr()), ctypes.c_void_p(wide[1].data_ptr()), 1, None):
        raise nse.Nse2dError(s.lib.nse2d_last_error().decode())
    out[0].copy_(wide[0])
    out[1].copy_(wide[1])
    return out


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        s = st["solver"]
        s.step(case["nsteps"], use_graph=True)
        return st["out"] if case["precision"] == 64 else _read32(s, st["wide"], st["out"])
    if kind == "run":
        s = st["solver"]
        reason = s.run(max_steps=case["nsteps"])
        t, dt, n, _ = s.time()
        return {"fields": st["out"], "reason": reason, "t": t, "dt": dt, "steps": n, "diag": s.diagnostics()}
    if kind == "closure":
        st["solver"].step(case["nsteps"], use_graph=True)
        return st["out"]
    if kind == "ensemble":
        st["ensemble"].step(case["nsteps"])
        if case["precision"] == 64:
            return st["out"]
        return [_read32(s, w, o) for s, w, o in zip(st["solvers"], st["wide"], st["out"])]
    if kind == "poisson":
        st["solver"].poisson_solve(st["w"], st["psi"])
        return st["psi"]
    if kind == "train":
        net = st["net"]
        loss = net.train_step(*st["fields"], 1e-5, idx=st["idx"], weight_decay=1e-4)
        return {"loss": loss, "grads": [net.get_grads(layer) for layer in range(net.layers)]}
    s = st["solver"]
    s.spectra_accumulate()
    kx, eu, ev, n = s.spectra()
    return {"diag": s.diagnostics(), "moments": s.row_moments(), "spectra": [kx, eu, ev], "samples": n}


def _step_work(Nx, Ny, real, steps):
    """omega and psi read and written once a step; the flops of the three stages (stencil ~70 a point, two real row transforms, a tridiagonal solve)."""
    n = Nx * Ny
    return {"bytes": 4.0 * real * n * steps, "flops": 3.0 * n * (70.0 + 5.0 * math.log2(Nx) + 10.0) * steps}


def _conv_flops(case, batch):
    h = case["hidden"]
    return 2.0 * 9.0 * (5 * h + 2 * h * h + h) * case["Nx"] * case["Ny"] * batch


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        w = [_step_work(c["Nx"], c["Ny"], 8 if c["precision"] == 64 else 4, case["nsteps"]) for c in _members(case, 0)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    Nx, Ny = case["Nx"], case["Ny"]
    n = Nx * Ny
    if kind in ("step", "run"):
        return _step_work(Nx, Ny, 8 if case["precision"] == 64 else 4, case["nsteps"])
    if kind == "poisson":
        return {"bytes": 16.0 * n, "flops": n * (5.0 * math.log2(Nx) + 10.0)}
    if kind == "closure":
        w = _step_work(Nx, Ny, 8, case["nsteps"])
        w["flops"] += 3 * case["nsteps"] * _conv_flops(case, 1)
        return w
    if kind == "train":
        return {"bytes": 40.0 * n * case["batch"], "flops": 3.0 * _conv_flops(case, case["batch"])}
    return {"bytes": 16.0 * n, "flops": n * (100.0 + 5.0 * math.log2(Nx))}


# ---- the same in 64 bits, in plain torch ----

class _Channel:
    """The mapped-grid channel: metrics, Poisson solve, wall closure, right-hand side, SSPRK(3,3) step."""

    def __init__(self, case):
        self.cfg = c = _cfg(case)
        Nx, Ny, b = c["Nx"], c["Ny"], c["beta"]
        t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=F64, device="cuda")  # noqa: E731
        self.Nx, self.Ny = Nx, Ny
        self.dx, self.de = LX / Nx, 2.0 / (Ny - 1)
        e = -1.0 + 2.0 * np.arange(Ny) / (Ny - 1)
        y = _y(Ny, b)
        an = np.tanh(b) * np.cosh(b * e) ** 2 / b if b > 0 else np.full(Ny, 1.0)
        ae = 0.5 * (an[:-1] + an[1:])
        dy = np.diff(y)
        self.nu = 2.0 / c["Reb"]
        self.dymin = float(np.min(dy))
        self.an, self.ae, self.dyh = t(an), t(ae), dy
        self.f = t(-c["F0"] * c["nforce"] * np.pi / 2.0 * np.cos(c["nforce"] * np.pi * (y + 1.0) / 2.0))[:, None]
        self.sub = np.zeros(Ny)
        self.sup = np.zeros(Ny)
        self.sub[1:-1] = an[1:-1] * ae[:-1] / self.de ** 2
        self.sup[1:-1] = an[1:-1] * ae[1:] / self.de ** 2
        k = torch.arange(Nx // 2 + 1, dtype=F64, device="cuda") * (2 * math.pi / LX)
        self.inv, self.cp = [], []
        cp = torch.zeros_like(k)
        for j in range(1, Ny - 1):
            den = -(self.sub[j] + self.sup[j]) - k * k - self.sub[j] * cp * (j > 1)
            cp = self.sup[j] / den
            self.inv.append(1.0 / den)
            self.cp.append(cp)

    def poisson(self, w):
        r = -torch.fft.rfft(w, dim=1)
        Ny = self.Ny
        r[Ny - 2, 0] -= self.sup[Ny - 2] * 2.0 * self.Nx
        d, out = torch.zeros_like(r[0]), []
        for j in range(1, Ny - 1):
            d = (r[j] - self.sub[j] * d) * self.inv[j - 1]
            out.append(d)
        x = torch.zeros_like(r)
        x[Ny - 1, 0] = 2.0 * self.Nx
        q = torch.zeros_like(r[0])
        for j in range(Ny - 2, 0, -1):
            q = torch.addcmul(out[j - 1], self.cp[j - 1].to(q.dtype), q, value=-1)
            x[j] = q
        return torch.fft.irfft(x, n=self.Nx, dim=1)

    def walls(self, w, psi):
        for j, j1, j2, d1, d2, pw in ((0, 1, 2, self.dyh[0], self.dyh[1], 0.0), (-1, -2, -3, self.dyh[-1], self.dyh[-2], 2.0)):
            A = 2.0 * (1.0 / (d1 * d1) + 1.0 / (d1 * d2))
            B = -2.0 * d1 / (d2 * (d1 + d2) ** 2)
            w[j] = -(A * (psi[j1] - pw) + B * (psi[j2] - pw))

    def rhs(self, psi, w):
        R = lambda a, s: torch.roll(a, -s, 1)  # noqa: E731
        a = self.an[1:-1, None]
        p, o = psi[1:-1], w[1:-1]
        pu, pd, ou, od = psi[2:], psi[:-2], w[2:], w[:-2]
        J1 = (R(p, 1) - R(p, -1)) * (ou - od) - (pu - pd) * (R(o, 1) - R(o, -1))
        J2 = R(p, 1) * (R(ou, 1) - R(od, 1)) - R(p, -1) * (R(ou, -1) - R(od, -1)) - pu * (R(ou, 1) - R(ou, -1)) + pd * (R(od, 1) - R(od, -1))
        J3 = -R(o, 1) * (R(pu, 1) - R(pd, 1)) + R(o, -1) * (R(pu, -1) - R(pd, -1)) + ou * (R(pu, 1) - R(pu, -1)) - od * (R(pd, 1) - R(pd, -1))
        J = -a * (J1 + J2 + J3) / (12.0 * self.dx * self.de)
        lap = (R(o, 1) - 2 * o + R(o, -1)) / self.dx ** 2 + a * (self.ae[1:, None] * (ou - o) - self.ae[:-1, None] * (o - od)) / self.de ** 2
        r = self.f - self.cfg["lin_drag"] * w
        r[1:-1] += self.nu * lap - J
        return r

    def dt(self, psi):
        v = (torch.roll(psi, -1, 1) - torch.roll(psi, 1, 1))[1:-1].abs() / (2 * self.dx)
        u = (self.an[1:-1, None] * (psi[2:] - psi[:-2])).abs() / (2 * self.de)
        um, vm = float(u.max()), float((v * self.an[1:-1, None]).max())
        adv = min(0.5 * self.dx / um if um > 0 else 1e30, 0.5 * self.de / vm if vm > 0 else 1e30)
        return min(self.cfg["dt_max"], adv, 0.25 / (self.nu * (1.0 / self.dx ** 2 + 1.0 / self.dymin ** 2)))

    def start(self, seed):
        w = _omega(self.Nx, self.Ny, self.cfg["beta"], seed)
        psi = self.poisson(w)
        self.walls(w, psi)
        return w, psi

    def step(self, w, psi, tau=None):
        dt = self.dt(psi)
        w0, wi = w, w
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
            r = self.rhs(psi, wi)
            if tau is not None:
                r = r - tau(wi, psi)
            wi = a * w0 + b * (wi + dt * r)
            psi = self.poisson(wi)
            self.walls(wi, psi)
        return wi, psi, dt

    def uv(self, psi):
        up, dn = torch.cat([psi[1:], psi[-1:]]), torch.cat([psi[:1], psi[:-1]])
        u = self.an[:, None] * (up - dn) / (2 * self.de)
        v = -(torch.roll(psi, -1, 1) - torch.roll(psi, 1, 1)) / (2 * self.dx)
        return u, v


def _params64(case, seed):
    """The weights of Cnn.init_params, as [cout, cin, 3, 3] in 64 bits."""
    rng = np.random.default_rng(seed)
    ch = [5] + [case["hidden"]] * 3 + [1]
    out = []
    for layer in range(4):
        ci, co = ch[layer], ch[layer + 1]
        bound = np.sqrt(6.0 / (9 * ci)) * (0.1 if layer == 3 else 1.0)
        w = rng.uniform(-bound, bound, (co, 9, ci)).astype(np.float32)
        out.append((torch.tensor(w, dtype=F64, device="cuda").reshape(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous(),
                    torch.zeros(co, dtype=F64, device="cuda")))
    return out


def _forward64(params, w, psi, u, v, y):
    s = _SCALES[0]
    x = torch.stack([w / s[0], psi / s[1], u / s[2], v / s[3], y[:, None].expand_as(w[0]).expand_as(w)], 1)
    for layer, (k, b) in enumerate(params):
        x = torch.nn.functional.pad(torch.cat([x[..., -1:], x, x[..., :1]], -1), (0, 0, 1, 1))
        x = torch.nn.functional.conv2d(x, k, b)
        if layer < 3:
            x = torch.nn.functional.gelu(x, approximate="tanh")
    return x[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for c in _members(case, seed):
            ch = _Channel(c)
            w, psi = ch.start(c["seed"])
            for _ in range(case["nsteps"]):
                w, psi, _ = ch.step(w, psi)
            out.append([w, psi])
        return out
    if kind == "train":
        params = [(k.requires_grad_(), b.requires_grad_()) for k, b in _params64(case, seed)]
        f = _fields(case, seed, case["batch"] + 3)
        idx = torch.tensor(np.random.default_rng(seed).permutation(case["batch"] + 3)[:case["batch"]].copy(), device="cuda")
        w, psi, u, v, tau = (a[idx] for a in f)
        y = torch.tensor(_y(case["Ny"], case["beta"]), dtype=F64, device="cuda")
        loss = ((_forward64(params, w, psi, u, v, y) - tau / _SCALES[1])[:, 1:-1] ** 2).mean()
        loss.backward()
        return {"loss": float(loss), "grads": [(k.grad.permute(0, 2, 3, 1).reshape(k.shape[0], 9, k.shape[1]).contiguous(), b.grad) for k, b in params]}
    ch = _Channel(case)
    if kind == "poisson":
        return ch.poisson(_omega(case["Nx"], case["Ny"], case["beta"], seed))
    w, psi = ch.start(seed)
    if kind == "sample":
        u, v = ch.uv(psi)
        wt = torch.full((ch.Nx // 2 + 1,), 2.0, dtype=F64, device="cuda")
        wt[0] = wt[-1] = 1.0
        E = [wt * torch.fft.rfft(a, dim=1).abs().square().sum(0) / (ch.Nx ** 2 * ch.Ny) for a in (u, v)]
        kx = torch.arange(ch.Nx // 2 + 1, dtype=F64, device="cuda") * (2 * math.pi / LX)
        return {"diag": None, "moments": torch.stack([u.sum(1), v.sum(1), (u * u).sum(1), (v * v).sum(1), (u * v).sum(1)]),
                "spectra": [kx] + E, "samples": None}
    tau = None
    if kind == "closure":
        params, y = _params64(case, seed), torch.tensor(_y(ch.Ny, case["beta"]), dtype=F64, device="cuda")

        def tau(wi, p):
            u, v = ch.uv(p)
            z = _forward64(params, wi[None], p[None], u[None], v[None], y)[0].mean(1, keepdim=True) * (0.25 * _SCALES[1])
            z[0] = z[-1] = 0.0
            return z
    t = 0.0
    for _ in range(case["nsteps"]):
        w, psi, dt = ch.step(w, psi, tau)
        t += dt
    if kind == "run":
        return {"fields": [w, psi], "reason": None, "t": t, "dt": dt, "steps": None, "diag": None}
    return [w, psi]
