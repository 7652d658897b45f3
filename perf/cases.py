"""The workloads of a user of the DUGKS engine, for timing and comparing builds of it.

Each case is one call sequence through the public Python binding (pydugks.Engine,
dugks_autograd) on a flow of this repository's configurations:

  flow "channel"  turbulent channel on the tanh mesh (workloads.channel_config)
       "laminar"  body-force channel on the uniform mesh (workloads.laminar_config)
       "box"      periodic Taylor-Green box (workloads.taylor_green_config)
  op   "run"      `steps` steps of the state in device memory (dg_step / dg_run)
       "gradient" kinetic-energy gradient with respect to the first state through
                  `steps` steps, checkpoints every `every` (dugks_autograd.run)
       "segment"  `steps` states recorded from a checkpoint and reversed by the adjoint
                  with a body-force field as control (dg_run_store, dg_adjoint_run,
                  dg_field_grad)
       "stats"    the diag.dat / profiles-2.dat values of a state (dg_stats_values)
       "monitored" host state in, `steps` steps each followed by a host read of the
                  conserved moments, host state out (dg_set_state, dg_moments, dg_get_state)

`exact` restates the step in double precision with plain torch.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "dugks-gpu_gb300"))

import dugks_autograd as da  # noqa: E402
import pydugks  # noqa: E402
import workloads  # noqa: E402

BYTES = {"fp64": 8, "fp32": 4, "fp16": 2, "bf16": 2}
U0 = 0.05  # amplitude of the periodic box


def _case(name, op, flow, precision, nx, ny, nz, steps=1, every=0, recon="trilinear"):
    return {"name": name, "op": op, "flow": flow, "precision": precision, "nx": nx, "ny": ny, "nz": nz,
            "steps": steps, "every": every, "recon": recon}


def listed():
    return [
        # one dg_step call per time step on the smallest grid, as the C++ driver's loop does
        _case("laminar-step-fp64", "run", "laminar", "fp64", 64, 32, 32, 1),
        # the same grid advanced in one dg_run call between two outputs
        _case("laminar-run-fp32", "run", "laminar", "fp32", 64, 32, 32, 16),
        # periodic box in the default precision
        _case("box-run-fp64", "run", "box", "fp64", 64, 64, 64, 2),
        # the benchmark channel in every precision form
        _case("channel-run-fp64", "run", "channel", "fp64", 128, 128, 256, 2),
        _case("channel-run-fp32", "run", "channel", "fp32", 128, 128, 256, 4),
        _case("channel-run-fp16", "run", "channel", "fp16", 128, 128, 256, 4),
        # sizes that fill neither a warp, a tile nor a wave
        _case("ragged-run-bf16", "run", "channel", "bf16", 101, 75, 149, 4),
        # the central-difference reconstruction on the stretched mesh
        _case("ragged-gradrecon-fp32", "run", "channel", "fp32", 97, 66, 130, 4, recon="gradient"),
        # initial-state gradient of the periodic box (forward, recomputation, adjoint)
        _case("box-gradient-fp32", "gradient", "box", "fp32", 64, 64, 64, 8, every=4),
        # one checkpoint segment of the force-field gradient on the adjoint channel
        _case("channel-segment-fp32", "segment", "channel", "fp32", 128, 96, 192, 8),
        # the statistics written every output interval
        _case("channel-stats-fp64", "stats", "channel", "fp64", 128, 128, 256, 0),
        # a host program that uploads its state, watches the moments and downloads the result
        _case("channel-monitored-fp64", "monitored", "channel", "fp64", 64, 64, 96, 4),
    ]


def draw(rng):
    op = rng.choice(["run"] * 6 + ["gradient", "segment", "stats", "monitored"])
    flow = {"gradient": "box", "segment": "channel"}.get(op) or rng.choice(["channel", "channel", "laminar", "box"])
    if op in ("gradient", "segment"):
        precision = rng.choice(["fp32", "fp32", "fp64"])
    else:
        precision = rng.choice(["fp64", "fp32", "fp16", "bf16"])
    top = 4.0e6 if op in ("run", "stats") else 1.0e6
    cells = math.exp(rng.uniform(math.log(8.0e3), math.log(top)))
    side = cells ** (1.0 / 3.0)
    nx = max(16, int(side * math.exp(rng.uniform(-0.5, 0.5))))
    ny = max(8, int(side * math.exp(rng.uniform(-0.5, 0.5))))
    nz = max(8, int(cells / (nx * ny)))
    nz = min(nz, int(top / (nx * ny)))
    recon = "gradient" if op == "run" and rng.random() < 0.2 else "trilinear"
    steps = 0 if op == "stats" else rng.choice([1, 2, 3, 4])
    if precision == "fp64" and cells > 1.0e6:
        steps = min(steps, 2)
    return {"op": op, "flow": flow, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "steps": steps,
            "every": rng.choice([2, 4]) if op == "gradient" else 0, "recon": recon}


# --- inputs ---------------------------------------------------------------------------------

def _config(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kw = dict(precision=case["precision"], recon=case["recon"])
    if case["flow"] == "channel":
        # wall resolution (cells per viscous length) of the Re_tau = 180 channel on 128 columns at any nx
        return workloads.channel_config(nx=nx, ny=ny, nz=nz, re_tau=180.0 * min(nx, 128) / 128, seed=seed % 100000,
                                        **kw)[0]
    if case["flow"] == "laminar":
        # Re_centre = 100 at centreline velocity 0.1 across nx cells
        visc = 0.0005 * nx
        return workloads.laminar_config(nx=nx, ny=ny, nz=nz, xwidth=nx, ywidth=ny, zwidth=nz, visc=f"{visc:.9g}",
                                        ambient_fz=f"{0.08 * visc / nx ** 2:.9g}", **kw)
    return workloads.taylor_green_config(n=nx, u0=U0, ny=ny, nz=nz, ywidth=ny, zwidth=nz, **kw)


def _lattice():
    c = torch.tensor(da._C, dtype=torch.float64, device="cuda")
    w = torch.tensor(da._W, dtype=torch.float64, device="cuda")
    return c, w


_CX, _CY, _CZ = ([row[p] for p in range(19)] for row in da._C)
_OPP = [0, 2, 1, 4, 3, 6, 5, 10, 9, 8, 7, 14, 13, 12, 11, 18, 17, 16, 15]


def _feq(rho, u):
    """Second-order equilibrium, (19, ...) for rho (...) and u (3, ...)."""
    c, w = _lattice()
    base = 1.0 - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    out = torch.empty((19,) + rho.shape, dtype=torch.float64, device="cuda") if not rho.requires_grad else None
    rows = []
    for p in range(19):
        eu = 3.0 * sum(float(c[a, p]) * u[a] for a in range(3))
        v = w[p] * rho * (base + eu + 0.5 * eu * eu)
        if out is None:
            rows.append(v)
        else:
            out[p] = v
    return torch.stack(rows) if out is None else out


def _start64(case, seed):
    """The box's or the laminar channel's seeded state (19, nz, ny, nx) in double precision: the
    flow of its configuration with a few seeded waves and a small non-equilibrium part."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device="cpu").manual_seed(seed)
    z, y, x = torch.meshgrid(*[(torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * (2 * math.pi / n)
                               for n in (nz, ny, nx)], indexing="ij")
    u = torch.zeros((3, nz, ny, nx), dtype=torch.float64, device="cuda")
    if case["flow"] == "box":
        u[0] = U0 * torch.sin(x) * torch.cos(y) * torch.cos(z)
        u[1] = -U0 * torch.cos(x) * torch.sin(y) * torch.cos(z)
    else:
        u[2] = 0.1 * torch.sin(0.5 * x)
    k = torch.randint(1, 4, (3, 4, 3), generator=g).tolist()
    ph = (torch.rand((3, 4), generator=g, dtype=torch.float64) * 2 * math.pi).tolist()
    for a in range(3):
        for m in range(4):
            kx = k[a][m][0] * (1.0 if case["flow"] == "box" else 0.5)
            u[a] += 0.004 * torch.sin(kx * x + k[a][m][1] * y + k[a][m][2] * z + ph[a][m])
    rho = 1.0 + 0.002 * torch.cos(x + ph[0][0]) * torch.sin(y + ph[0][1]) * torch.cos(z + ph[0][2])
    f = _feq(rho, u)
    noise = torch.rand((nz, ny, nx), generator=g, dtype=torch.float64).cuda() - 0.5
    for p in range(19):
        f[p] *= 1.0 + 1e-3 * torch.roll(noise, p, 2)
    return f


def _field(case, seed):
    """Seeded body-force field, a few per cent of the channel's mean force."""
    r = np.random.default_rng(seed + 77)
    return 2.0e-7 * r.standard_normal((case["nz"], case["ny"], case["nx"]))


class _Raw:
    """A CUDA array interface over the engine's buffer; holds the engine as long as a tensor uses it."""

    def __init__(self, eng, ptr, n, typestr):
        self.owner = eng
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (int(ptr), False),
                                         "strides": None, "version": 3}


def _view(eng):
    """(19, nz, ny, nx) view of the engine's own state, in its storage type."""
    p = eng.info.precision
    ts = ("<f8", "<f4", "<f2", "<i2")[p]
    t = torch.as_tensor(_Raw(eng, eng.device_ptr(pydugks.DG_BUF_F), eng.soa_len, ts), device="cuda")
    return da.soa_view(eng, t.view(torch.bfloat16) if p == 3 else t)


def prepare(case, seed):
    eng = pydugks.Engine(_config(case, seed))
    s = {"case": case, "eng": eng, "istep": 1}
    if case["flow"] != "channel":
        f = _start64(case, seed)
        if case["precision"] in ("fp64", "fp32"):
            t = da.from_dump_order(eng, f.permute(1, 2, 3, 0))
            eng.set_state_device(t.data_ptr())
            s["f0"] = t
        else:
            eng.set_state(f.permute(1, 2, 3, 0).contiguous().cpu().numpy())
        torch.cuda.synchronize()
    if case["op"] == "segment":
        eng.set_force_field(2, _field(case, seed))
        s["f0"] = da.empty_state(eng)
        eng.get_state_device(s["f0"].data_ptr())
        s["states"] = torch.zeros((case["steps"], eng.soa_len), dtype=s["f0"].dtype, device="cuda")
        s["lam0"] = torch.zeros(eng.soa_len, dtype=s["f0"].dtype, device="cuda")
        da.soa_view(eng, s["lam0"]).copy_(_lam64(case, seed))
        s["lam"] = torch.empty_like(s["lam0"])
    elif case["op"] == "gradient":
        s["f0"].requires_grad_(True)
    elif case["op"] == "monitored":
        s["host"] = eng.get_state()
    if case["op"] in ("run", "stats"):
        s["out"] = _view(eng)
    torch.cuda.synchronize()
    return s


def _lam64(case, seed):
    g = torch.Generator(device="cpu").manual_seed(seed + 5)
    shape = (19, case["nz"], case["ny"], case["nx"])
    return torch.rand(shape, generator=g, dtype=torch.float32).cuda().double() - 0.5


def run(s):
    case, eng = s["case"], s["eng"]
    op, n = case["op"], case["steps"]
    if op == "run":
        if n == 1:
            eng.step(s["istep"])
        else:
            eng.run(s["istep"], n)
        s["istep"] += n
        return {"f": s["out"]}
    if op == "gradient":
        fn = da.run(s["f0"], eng, 1, n, every=case["every"])
        J = da.kinetic_energy(eng, fn)
        (g,) = torch.autograd.grad(J, s["f0"])
        return {"J": J.detach(), "f": da.soa_view(eng, fn.detach()), "grad": da.soa_view(eng, g)}
    if op == "segment":
        eng.set_state_device(s["f0"].data_ptr())
        stride = s["states"].stride(0) * s["states"].element_size()
        s["lam"].copy_(s["lam0"])
        eng.run_store(1, n, s["states"].data_ptr(), stride)
        eng.adjoint_run(1, n, s["states"].data_ptr(), stride, s["lam"].data_ptr())
        return {"lam": da.soa_view(eng, s["lam"]), "dphi": eng.field_grad(reset=True),
                "last": da.soa_view(eng, s["states"][n - 1])}
    if op == "stats":
        diag, prof = eng.stats_values()
        return {"diag": diag, "prof": prof}
    eng.set_state(s["host"])
    mom = []
    for k in range(n):
        eng.step(1 + k)
        mom.append(eng.moments())
    return {"f": eng.get_state(), "moments": np.stack(mom)}


def work(case):
    """Per step and cell: the state read once and written once (the adjoint: state and adjoint read,
    adjoint written); about 900 operations for the step, twice that for its adjoint."""
    cells = case["nx"] * case["ny"] * case["nz"]
    b, n = 19.0 * BYTES[case["precision"]] * cells, case["steps"]
    op = case["op"]
    if op == "stats":
        return {"bytes": b, "flops": 70.0 * cells}
    if op == "run":
        return {"bytes": 2 * b * n, "flops": 900.0 * cells * n}
    if op == "monitored":
        return {"bytes": 2 * 152.0 * cells + 3 * b * n, "flops": 940.0 * cells * n}
    # forward, recomputation (gradient), adjoint
    sweeps = 2 if op == "gradient" else 1
    return {"bytes": (2 * sweeps + 3) * b * n, "flops": (900.0 * sweeps + 1800.0) * cells * n}


# --- the step restated in double precision ---------------------------------------------------

class _Setup:
    """Mesh, coefficients and start of a case from its configuration text alone."""

    def __init__(self, case, seed):
        kv = dict(line.split("=", 1) for line in _config(case, seed).splitlines() if "=" in line)
        real = {k: float(np.float32(float(kv[k]))) for k in ("xwidth", "ywidth", "zwidth", "CFL", "visc", "ambient_fx",
                                                             "ambient_fy", "ambient_fz")}
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.n, self.walls, self.recon = (nx, ny, nz), kv["periods_x"] == "0", case["recon"]
        self.width = tuple(real[k] for k in ("xwidth", "ywidth", "zwidth"))
        self.F = [real["ambient_fx"], real["ambient_fy"], real["ambient_fz"]]
        self.dx, self.dy, self.dz = self.width[0] / nx, self.width[1] / ny, self.width[2] / nz
        self.tanh = kv.get("mesh", "uniform") == "tanh"
        if self.tanh:
            a, L = float(kv["mesh_alpha"]), float(kv["xwidth"])
            eta = -1.0 + 2.0 * np.arange(nx + 1) / nx
            xf = L / (2 * a) * np.tanh(eta * 0.5 * (math.log(1 + a) - math.log(1 - a))) + 0.5 * L
        else:
            xf, L = self.dx * np.arange(nx + 1), self.width[0]
        xc, dxx = np.zeros(nx + 2), np.zeros(nx + 2)
        xc[1:-1], dxx[1:-1] = 0.5 * (xf[1:] + xf[:-1]), xf[1:] - xf[:-1]
        xc[0], xc[-1], dxx[0], dxx[-1] = -xc[1], 2 * L - xc[nx], dxx[1], dxx[nx]
        self.xc, self.dxx = xc, dxx
        self.dt = real["CFL"] * (dxx[1] if self.tanh else self.dx) / math.sqrt(2.0)
        self.hdt = h = 0.5 * self.dt
        tau = real["visc"] * 3.0
        self.bw = (3 * tau * h / (2 * tau + self.dt), (2 * tau - h) / (2 * tau + self.dt), 3 * h / (2 * tau + self.dt))
        self.fw = (tau * h / (2 * tau + h), 2 * tau / (2 * tau + h), h / (2 * tau + h))
        self.phi = None
        # the engine's own start, from which the 16-bit forms take their scales
        if case["flow"] == "channel":
            self.f0 = self.own = self._channel_start(kv)
        else:
            self.f0 = _start64(case, seed)
            self.own = self._uniform_start(case)
        if case["op"] == "segment":
            self.phi = torch.from_numpy(_field(case, seed)).cuda()

    def _uniform_start(self, case):
        nx, ny, nz = self.n
        u = torch.zeros((3, nz, ny, nx), dtype=torch.float64, device="cuda")
        rho = torch.ones((nz, ny, nx), dtype=torch.float64, device="cuda")
        if case["flow"] == "laminar":
            u[2] = 0.1
        else:
            z, y, x = torch.meshgrid(*[(torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * (2 * math.pi / n)
                                       for n in (nz, ny, nx)], indexing="ij")
            rho = 1.0 + 3.0 * U0 * U0 / 16 * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2)
            u[0] = U0 * torch.sin(x) * torch.cos(y) * torch.cos(z)
            u[1] = -U0 * torch.cos(x) * torch.sin(y) * torch.cos(z)
        return _feq(rho, u)

    def _channel_start(self, kv):
        """Poiseuille profile, seeded uniform perturbations (splitmix64) and near-wall streaks."""
        nx, ny, nz = self.n
        ub, re_tau, seed = float(kv["ub"]), float(kv["re_tau"]), int(kv["seed"])
        cell = np.arange(nx * ny * nz, dtype=np.uint64)
        x = torch.from_numpy(self.xc[1:-1]).cuda()
        y = (torch.arange(ny, dtype=torch.float64, device="cuda") + 0.5) * self.dy
        u = torch.empty((3, nz, ny, nx), dtype=torch.float64, device="cuda")
        for a in range(3):
            with np.errstate(over="ignore"):
                z = np.uint64((seed * 0xD1B54A32D192ED03) & (2 ** 64 - 1)) + cell * np.uint64(3) + np.uint64(a)
                z = z + np.uint64(0x9E3779B97F4A7C15)
                z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
                z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
                z = z ^ (z >> np.uint64(31))
            r = (z >> np.uint64(11)).astype(np.float64) * (2.0 / 9007199254740992.0) - 1.0
            u[a] = torch.from_numpy(0.1 * ub * r).cuda().view(nz, ny, nx)
        W = self.width[0]
        eta = x / W
        et = torch.minimum(x, W - x) * (re_tau / (0.5 * W)) / 10.0
        u[2] += 6.0 * ub * eta * (1 - eta)
        u[2] += 0.05 * ub * torch.sin(2 * math.pi * 4 * y / self.width[1]).view(1, ny, 1) * (et * torch.exp(1 - et))
        return _feq(torch.ones((nz, ny, nx), dtype=torch.float64, device="cuda"), u)

    # --- step ---
    def _force(self, phi):
        return [self.F[0], self.F[1], self.F[2] if phi is None else self.F[2] + phi]

    def _relaxed(self, f, rho, u, F, w0, w1, w2):
        """w1 f + (w2 + 3 w0 F.(c - u)) feq(rho, u) for every population."""
        fu = F[0] * u[0] + F[1] * u[1] + F[2] * u[2]
        fe = _feq(rho, u)
        rows = []
        for p in range(19):
            cf = _CX[p] * F[0] + _CY[p] * F[1] + _CZ[p] * F[2]
            rows.append(w1 * f[p] + (w2 + 3 * w0 * (cf - fu)) * fe[p])
        return torch.stack(rows)

    @staticmethod
    def _moments(f):
        rho = f.sum(0)
        j = [sum(c[p] * f[p] for p in range(19) if c[p]) for c in (_CX, _CY, _CZ)]
        return rho, j

    def _shift_force(self, j, rho, F, h):
        return torch.stack([j[a] / rho + h * F[a] for a in range(3)])

    def _pad(self, a):
        """One ghost layer around (..., nz, ny, nx): walls (extrapolated) or periodic in x, periodic in y, z."""
        if self.walls:
            q0, q1 = 2.0, 2.0
            if self.tanh:
                xc, n = self.xc, self.n[0]
                q0 = (xc[2] - xc[0]) / (xc[2] - xc[1])
                q1 = (xc[n + 1] - xc[n - 1]) / (xc[n] - xc[n - 1])
            lo = q0 * a[..., :1] + (1 - q0) * a[..., 1:2]
            hi = q1 * a[..., -1:] + (1 - q1) * a[..., -2:-1]
        else:
            lo, hi = a[..., -1:], a[..., :1]
        a = torch.cat([lo, a, hi], -1)
        a = torch.cat([a[..., -1:, :], a, a[..., :1, :]], -2)
        return torch.cat([a[..., -1:, :, :], a, a[..., :1, :, :]], -3)

    def _faces(self, fb, ax):
        """Face values (19, nz, ny, nfaces...) of orientation ax from the padded f-bar-plus."""
        h, T = self.hdt, lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
        dxx, xc = self.dxx, self.xc
        nx, ny, nz = self.n
        if not self.tanh:
            dxx = np.full(nx + 2, self.dx)
        # the two cells across the face: slices along each axis of the padded array
        lo, hi, mid = {0: slice(0, nx + 1), 1: slice(1, ny + 1), 2: slice(1, nz + 1)}, {0: slice(1, nx + 2), 1: slice(
            2, ny + 2), 2: slice(2, nz + 2)}, {0: slice(1, nx + 1), 1: slice(1, ny + 1), 2: slice(1, nz + 1)}
        sh = lambda s, d: slice(s.start + d, s.stop + d)  # noqa: E731

        def at(g, side, dx=0, dy=0, dz=0):
            s = [mid[0], mid[1], mid[2]]
            s[ax] = hi[ax] if side else lo[ax]
            s = [sh(s[0], dx), sh(s[1], dy), sh(s[2], dz)]
            return g[s[2], s[1], s[0]]

        rows = []
        for p in range(19):
            g, c = fb[p], (_CX[p], _CY[p], _CZ[p])
            if self.recon == "gradient":
                rows.append(self._grad_face(g, c, ax, at, T))
                continue

            def value(side):
                """Transverse characteristic interpolation at the cells on one side."""
                def alongx(dy, dz):
                    if ax == 0 or c[0] == 0:
                        return at(g, side, 0, dy, dz)
                    i = np.arange(1, nx + 1)
                    t = T(h / (0.5 * dxx[i] + 0.5 * dxx[i - c[0]]))
                    return (1 - t) * at(g, side, 0, dy, dz) + t * at(g, side, -c[0], dy, dz)

                def alongy(dz):
                    if ax == 1 or c[1] == 0:
                        return alongx(0, dz)
                    t = h / self.dy
                    return (1 - t) * alongx(0, dz) + t * alongx(-c[1], dz)

                if ax == 2 or c[2] == 0:
                    return alongy(0)
                t = h / self.dz
                return (1 - t) * alongy(0) + t * alongy(-c[2])

            if p == 0:
                m = 0.5
            elif ax == 0:
                m = T((dxx[:-1] / 2 - h * c[0]) / (0.5 * dxx[:-1] + 0.5 * dxx[1:]))
            else:
                d = self.dy if ax == 1 else self.dz
                m = (d / 2 - h * c[ax]) / d
            rows.append((1 - m) * value(0) + m * value(1))
        return torch.stack(rows)

    def _grad_face(self, g, c, ax, at, T):
        """Mean across the face less hdt (c . gradient), central differences."""
        nx, dy, dz, xc, dxx = self.n[0], self.dy, self.dz, self.xc, self.dxx
        lam = 0.5
        if ax == 0 and self.tanh:
            lam = T(0.5 * dxx[:-1] / (xc[1:] - xc[:-1]))

        def mean(dx=0, dy_=0, dz_=0):
            a, b = at(g, 0, dx, dy_, dz_), at(g, 1, dx, dy_, dz_)
            return a + lam * (b - a)

        jump = at(g, 1) - at(g, 0)
        m = mean()
        if ax == 0:
            gx = jump * (T(1.0 / (xc[1:] - xc[:-1])) if self.tanh else 1.0 / self.dx)
        elif self.tanh:
            i = np.arange(1, nx + 1)
            hm, hp = xc[i] - xc[i - 1], xc[i + 1] - xc[i]
            gx = (T(-hp / (hm * (hp + hm))) * mean(dx=-1) + T((hp - hm) / (hp * hm)) * m
                  + T(hm / (hp * (hp + hm))) * mean(dx=1))
        else:
            gx = (mean(dx=1) - mean(dx=-1)) / (2 * self.dx)
        gy = jump / dy if ax == 1 else (mean(dy_=1) - mean(dy_=-1)) / (2 * dy)
        gz = jump / dz if ax == 2 else (mean(dz_=1) - mean(dz_=-1)) / (2 * dz)
        return m - self.hdt * (c[0] * gx + c[1] * gy + c[2] * gz)

    def step(self, f, phi=None):
        nx, ny, nz = self.n
        rho, j = self._moments(f)
        F = self._force(phi)
        fb = self._relaxed(f, rho, self._shift_force(j, rho, F, self.hdt), F, *self.bw)
        g = self._pad(fb)
        out = (4.0 / 3.0) * fb - (1.0 / 3.0) * f
        for ax, cs in enumerate((_CX, _CY, _CZ)):
            v = self._faces(g, ax)
            if ax == 0 and self.walls:
                rows = []
                for p in range(19):
                    col = v[p]
                    if cs[p] > 0:
                        col = torch.cat([v[_OPP[p]][..., :1], col[..., 1:]], -1)
                    elif cs[p] < 0:
                        col = torch.cat([col[..., :-1], v[_OPP[p]][..., -1:]], -1)
                    rows.append(col)
                v = torch.stack(rows)
            pf = phi
            if phi is not None:
                if ax == 0:
                    e = torch.cat([phi[..., :1] if self.walls else phi[..., -1:], phi,
                                   phi[..., -1:] if self.walls else phi[..., :1]], -1)
                    pf = 0.5 * (e[..., :-1] + e[..., 1:])
                else:
                    pf = 0.5 * (phi + torch.roll(phi, -1, 1 if ax == 1 else 0))
            rho, j = self._moments(v)
            F = self._force(pf)
            flux = self._relaxed(v, rho, self._shift_force(j, rho, F, 0.5 * self.hdt), F, *self.fw)
            if ax == 0:
                dxx = self.dxx[1:-1] if self.tanh else np.full(nx, self.dx)
                d = (flux[..., 1:] - flux[..., :-1]) * torch.from_numpy(self.dt / dxx).cuda()
            else:
                dim, h = (2, self.dy) if ax == 1 else (1, self.dz)
                d = (flux - torch.roll(flux, 1, dim)) * (self.dt / h)
            out = out - torch.stack([float(cs[p]) * d[p] for p in range(19)])
        return out

    def reverse(self, f, lam, phi=None):
        """(dS/df)^T lam and (dS/dphi)^T lam at the state f."""
        with torch.enable_grad():
            x = f.detach().requires_grad_(True)
            q = phi.detach().requires_grad_(True) if phi is not None else None
            y = self.step(x, q)
            got = torch.autograd.grad(y, [x] if q is None else [x, q], grad_outputs=lam)
        return got[0], (got[1] if q is not None else None)


def exact(case, seed):
    op, n = case["op"], case["steps"]
    if op in ("gradient", "segment") and case["nx"] * case["ny"] * case["nz"] * n > 1.0e7 and op == "gradient":
        return None
    S = _Setup(case, seed)
    f = S.f0
    if op == "stats":
        return _exact_stats(S, f)
    if op == "run":
        with torch.no_grad():
            for _ in range(n):
                f = S.step(f)
            if case["precision"] in ("fp16", "bf16"):
                w = torch.tensor(da._W, dtype=torch.float64, device="cuda").view(19, 1, 1, 1)
                scale = w * ((S.own - w).abs().amax((1, 2, 3), keepdim=True) / w).clamp(min=1e-3)
                f = (f - w) / scale
        return {"f": f}
    if op == "monitored":
        mom = []
        with torch.no_grad():
            for _ in range(n):
                f = S.step(f)
                rho, j = S._moments(f)
                mom.append([float(v.sum()) for v in (rho, *j)])
        return {"f": f.permute(1, 2, 3, 0).contiguous().cpu().numpy(), "moments": np.array(mom)}
    states = [f]
    with torch.no_grad():
        for _ in range(n if op == "gradient" else n - 1):
            states.append(S.step(states[-1], S.phi))
    if op == "segment":
        lam, dphi = _lam64(case, seed), torch.zeros_like(S.phi)
        for f in reversed(states):
            lam, d = S.reverse(f, lam, S.phi)
            dphi += d
        return {"lam": lam, "dphi": dphi.cpu().numpy(), "last": states[-1]}
    fn = states.pop().requires_grad_(True)
    rho, j = S._moments(fn)
    J = 0.5 * sum((a * a / rho) for a in j).sum()
    (lam,) = torch.autograd.grad(J, fn)
    for f in reversed(states):
        lam, _ = S.reverse(f, lam)
    return {"J": J.detach(), "f": fn.detach(), "grad": lam}


def _exact_stats(S, f):
    rho, j = S._moments(f)
    u = S._shift_force(j, rho, S.F, S.hdt)
    q = torch.stack([rho, u[0], u[1], u[2]])
    diag = torch.cat([q.mean((1, 2, 3)), q.amin((1, 2, 3)), q.amax((1, 2, 3))])
    m = u.mean((1, 2))                                     # (3, nx)
    cov = [(u[a] * u[b]).mean((0, 1)) - m[a] * m[b] for a, b in ((0, 2), (0, 1), (1, 2), (0, 0), (1, 1), (2, 2))]
    return {"diag": diag.cpu().numpy(), "prof": torch.stack([*m, *cov], 1).cpu().numpy()}


if __name__ == "__main__":
    for c in listed():
        print(c)
    print(draw(random.Random(0)))
