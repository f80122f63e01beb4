"""Workloads of this framework, as a program that uses it runs them.

Each case goes through public entry points: the 2D Crank-Nicolson engine and
its gradient, the 3D engine and its gradient (plain and learned
preconditioner), multislice in 2D and 3D with its autograd functions, the
space-time (PiT) solve and a training step of the learned preconditioner.
``listed()`` are the cases themselves, ``draw()`` gives further ones of the
same ranges, ``prepare()`` makes what a program holds before the call,
``run()`` is one call, ``work()`` what a call cannot do without, and
``exact()`` the same results in complex128 with plain torch operations.

Index fields are ``1 - dn`` for the paraxial solvers and ``1 + dn`` for
multislice (the two models' sign conventions), probes are Gaussians at scan
positions, lengths are in pixels of size 1.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from thick_ptycho_b200 import heads
from thick_ptycho_b200.cn2d import CN2D
from thick_ptycho_b200.cn3d import CN3D, PWEGradient3D
from thick_ptycho_b200.geometry import SimulationGeometry
from thick_ptycho_b200.gradient import PWEFunction, PWEGradient2D
from thick_ptycho_b200.learned import LearnedPreconditioner, default_kappa
from thick_ptycho_b200.ms2d import MS2D, MSFunction
from thick_ptycho_b200.ms3d import MS3D, MS3DFunction
from thick_ptycho_b200.pit import PiT2D

C64, C128 = torch.complex64, torch.complex128


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest forward simulation: 32 scan positions, exit waves and far field
        {"name": "2d-forward-256", "kind": "cn2d", "n": 256, "nz": 128, "probes": 32, "mode": "forward",
         "bc": "impedance", "full": False, "single": False, "wave": 0.5, "dz": 1.0},
        # simulation keeping the whole field, on the odd grids that an even scan step gives;
        # the index held as n - 1 in complex64
        {"name": "2d-field-odd-1201", "kind": "cn2d", "n": 1201, "nz": 600, "probes": 100, "mode": "forward",
         "bc": "neumann", "full": True, "single": True, "wave": 0.5, "dz": 1.0},
        # reconstruction gradient of the large 2D scan
        {"name": "2d-gradient-2048", "kind": "cn2d_grad", "n": 2048, "nz": 1024, "probes": 512, "bc": "impedance",
         "checkpoint": "none", "wave": 0.5, "dz": 1.0},
        # the autograd function inside a user's own loss, with sqrt checkpointing
        {"name": "2d-autograd-1024-sqrt", "kind": "cn2d_autograd", "n": 1024, "nz": 512, "probes": 256,
         "bc": "impedance", "checkpoint": "sqrt", "wave": 0.5, "dz": 1.0},
        # 3D simulation on a ragged grid with few probes, field kept
        {"name": "3d-forward-ragged-90x75", "kind": "cn3d", "nx": 90, "ny": 75, "nz": 48, "probes": 9,
         "mode": "forward", "bc": "dirichlet", "wave": 0.5, "dz": 1.0},
        # 3D gradient at full depth with the plain preconditioner
        {"name": "3d-gradient-256", "kind": "cn3d_grad", "nx": 256, "ny": 256, "nz": 256, "probes": 64,
         "bc": "impedance", "learned": False, "wave": 0.5, "dz": 1.0},
        # one gradient of a 3D reconstruction with the learned preconditioner in both marches
        {"name": "3d-gradient-192-learned", "kind": "cn3d_grad", "nx": 192, "ny": 192, "nz": 96, "probes": 64,
         "bc": "impedance", "learned": True, "wave": 0.5, "dz": 1.0},
        # multislice exit waves and their gradient, 2D
        {"name": "2d-multislice-2048", "kind": "ms2d", "n": 2048, "nz": 1024, "probes": 64, "wave": 0.5, "dz": 1.0},
        # multislice exit waves and their gradient, 3D
        {"name": "3d-multislice-256", "kind": "ms3d", "nx": 256, "ny": 256, "nz": 256, "probes": 64, "wave": 0.5,
         "dz": 1.0},
        # space-time GMRES of a whole scan
        {"name": "pit-256", "kind": "pit", "n": 256, "nz": 128, "probes": 32, "bc": "impedance", "wave": 0.5, "dz": 1.0},
        # one training step of the learned preconditioner: a batch of slices, all their probes
        {"name": "cnn-train-step-256", "kind": "cnn", "nx": 256, "ny": 256, "batch": 4, "probes": 16},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _plannable(rng, lo, hi):
    """A length 2^a 3^b 5^c between lo and hi, near a log-uniform draw."""
    n = _logint(rng, lo, hi)
    for d in range(n):
        for m in (n - d, n + d):
            if lo <= m <= hi and heads.fft_plannable(m):
                return m
    return lo


def draw(rng):
    kind = rng.choice(["cn2d", "cn2d", "cn2d_grad", "cn2d_autograd", "cn3d", "cn3d_grad", "cn3d_grad", "ms2d", "ms3d",
                       "pit", "cnn"])
    wave, dz = round(rng.uniform(0.4, 0.7), 3), rng.choice([0.5, 1.0, 1.0, 1.5])
    optics = {"wave": wave, "dz": dz}
    bc = rng.choice(["impedance", "impedance", "neumann", "dirichlet"])
    if kind == "cn2d":
        # the team sizes are as likely as all others together
        n = rng.choice([512, 1024, 2048]) if rng.random() < 0.5 else _logint(rng, 96, 2048)
        return {"kind": kind, "n": n, "nz": _logint(rng, 48, 1024), "probes": _logint(rng, 8, 256),
                "mode": rng.choice(["forward", "forward", "adjoint", "adjoint_exact"]),
                "bc": rng.choice([bc, "impedance2"]), "full": rng.random() < 0.5, "single": rng.random() < 0.5, **optics}
    if kind in ("cn2d_grad", "cn2d_autograd"):
        # loss_and_grad takes plannable lengths (its far field), the autograd function any
        n = (rng.choice([512, 1024, 2048]) if rng.random() < 0.5 else
             _plannable(rng, 128, 2048) if kind == "cn2d_grad" else _logint(rng, 96, 2048))
        return {"kind": kind, "n": n, "nz": _logint(rng, 64, 1024), "probes": _logint(rng, 16, 512), "bc": bc,
                "checkpoint": rng.choice(["none", "none", "sqrt"]), **optics}
    if kind == "cn3d":
        nx = rng.choice([64, 128, 192, 256]) if rng.random() < 0.4 else _logint(rng, 40, 200)
        ny = nx if rng.random() < 0.5 else _logint(rng, 40, 200)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": _logint(rng, 24, 128), "probes": _logint(rng, 4, 64),
                "mode": rng.choice(["forward", "forward", "adjoint"]), "bc": bc, **optics}
    if kind == "cn3d_grad":
        learned = rng.random() < 0.3
        nx = rng.choice([64, 128, 192, 256]) if rng.random() < 0.6 else _plannable(rng, 48, 240)
        return {"kind": kind, "nx": nx, "ny": nx, "nz": _logint(rng, 24, 128), "probes": _logint(rng, 4, 64),
                "bc": bc, "learned": learned, **optics}
    if kind == "ms2d":
        return {"kind": kind, "n": _plannable(rng, 128, 2048), "nz": _logint(rng, 64, 1024),
                "probes": _logint(rng, 8, 256), **optics}
    if kind == "ms3d":
        nx = rng.choice([64, 128, 256]) if rng.random() < 0.6 else _plannable(rng, 48, 256)
        return {"kind": kind, "nx": nx, "ny": nx if rng.random() < 0.6 else _plannable(rng, 48, 256),
                "nz": _logint(rng, 24, 256), "probes": _logint(rng, 4, 64), **optics}
    if kind == "pit":
        return {"kind": kind, "n": _logint(rng, 96, 1024), "nz": _logint(rng, 48, 512), "probes": _logint(rng, 4, 32),
                "bc": rng.choice(["impedance", "neumann"]), **optics}
    return {"kind": kind, "nx": _logint(rng, 48, 256), "ny": _logint(rng, 48, 256), "batch": rng.choice([1, 2, 4]),
            "probes": _logint(rng, 4, 32)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _noise(shape, g):
    """Complex standard normal, complex64."""
    return torch.randn(*shape, 2, generator=g, device="cuda").view(torch.float32).contiguous().view(C64).squeeze(-1)


def _dn_2d(n, nz, g):
    """Smooth blobs of |dn| <= 1e-3, a few to a few tens of pixels wide, with weak absorption."""
    coarse = torch.randn(1, 1, max(4, n // 24), max(4, nz // 24), generator=g, device="cuda", dtype=torch.float64)
    dn = torch.nn.functional.interpolate(coarse, size=(n, nz), mode="bicubic", align_corners=False)[0, 0]
    return (dn * (1e-3 / dn.abs().max())).to(C128) + 1e-5j


def _dn_3d(nx, ny, nz, g):
    """Homogeneous bodies of dn up to 5e-4 (a thresholded smooth random field), with weak absorption."""
    size = [max(3, m // 12) for m in (nx, ny, nz)]
    coarse = torch.randn(1, 1, *size, generator=g, device="cuda")
    s = torch.nn.functional.interpolate(coarse, size=(nx, ny, nz), mode="trilinear", align_corners=False)[0, 0]
    dn = torch.where(s > 0.6, 5e-4, torch.where(s > 0.3, 2e-4, 0.0)).to(torch.float64)
    return dn.to(C128) + 1e-6j


def _probes_1d(n, count, g):
    x = torch.arange(n, device="cuda", dtype=torch.float64)[None]
    c = n * (0.2 + 0.6 * (torch.arange(count, device="cuda", dtype=torch.float64) + 0.5) / count)
    c = (c + torch.rand(count, generator=g, device="cuda", dtype=torch.float64))[:, None]
    return torch.exp(-((x - c) ** 2) / 64.0).to(C64)


def _probes_2d(nx, ny, count, g):
    """(count, nx*ny), row-major with nx rows."""
    side = math.ceil(math.sqrt(count))
    i = torch.arange(count, device="cuda")
    jit = torch.rand(count, 2, generator=g, device="cuda", dtype=torch.float64)
    cx = nx * (0.3 + 0.4 * ((i // side) + 0.5) / side) + jit[:, 0]
    cy = ny * (0.3 + 0.4 * ((i % side) + 0.5) / side) + jit[:, 1]
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[None]
    y = torch.arange(ny, device="cuda", dtype=torch.float64)[None]
    w2 = (0.047 * min(nx, ny)) ** 2 + 4.0
    gx, gy = torch.exp(-((x - cx[:, None]) ** 2) / w2), torch.exp(-((y - cy[:, None]) ** 2) / w2)
    return (gx[:, :, None] * gy[:, None, :]).reshape(count, nx * ny).to(C64)


def _amplitude(far, g):
    """Measured amplitudes: brighter than the free-space far field, with 10 % spread."""
    a = far.abs().to(torch.float64)
    return 1.25 * a * (1 + 0.1 * torch.rand(a.shape, generator=g, device="cuda", dtype=torch.float64))


def _inputs(c, seed):
    """The tensors of a case, from the seed alone."""
    g, kind = _gen(seed), c["kind"]
    if kind in ("cn2d", "cn2d_grad", "cn2d_autograd", "pit"):
        n, nz, P = c["n"], c["nz"], c["probes"]
        field = 1 - _dn_2d(n, nz, g)
        probes = _probes_1d(n, P, g)
        if kind == "cn2d_autograd" or c.get("single"):
            field = (field - 1).to(C64)  # n - 1
        s = {"field": field, "probes": probes}
        if kind == "cn2d_grad":
            s["amplitude"] = _amplitude(torch.fft.fft(probes, dim=-1), g)
        if kind == "cn2d_autograd":
            s["upstream"] = _noise((P, n), g) * probes.abs()
        return s
    if kind in ("cn3d", "cn3d_grad"):
        nx, ny, nz, P = c["nx"], c["ny"], c["nz"], c["probes"]
        # the engine's vectors run along ny blocks of nx
        field = (1 - _dn_3d(ny, nx, nz, g)).reshape(nx * ny, nz)
        s = {"field": field, "probes": _probes_2d(ny, nx, P, g)}
        if kind == "cn3d_grad":
            far = torch.fft.fft2(s["probes"].reshape(P, nx, ny))
            s["amplitude"] = _amplitude(far, g).reshape(P, nx * ny)
        return s
    if kind == "ms2d":
        s = {"field": 1 + _dn_2d(c["n"], c["nz"], g), "probes": _probes_1d(c["n"], c["probes"], g)}
        s["upstream"] = _noise((c["probes"], c["n"]), g) * s["probes"].abs()
        return s
    if kind == "ms3d":
        nx, ny, P = c["nx"], c["ny"], c["probes"]
        s = {"field": (1 + _dn_3d(nx, ny, c["nz"], g)).reshape(nx * ny, -1), "probes": _probes_2d(nx, ny, P, g)}
        s["upstream"] = _noise((P, nx * ny), g) * s["probes"].abs()
        return s
    nx, ny, B, V = c["nx"], c["ny"], c["batch"], c["batch"] * c["probes"]
    diag = (-1j * 2 * math.pi * (_dn_3d(B, ny, nx, g) * -1)).reshape(B, nx * ny).to(C64)
    z = _noise((V, nx * ny), g)
    target = z + 0.01 * _noise((V, nx * ny), g)
    scale = torch.full((V,), 1.0 / (V * nx * ny * 2e-4), device="cuda")
    return {"diag": diag, "z": z, "target": target, "scale": scale}


def _k(c):
    return 2 * math.pi / c["wave"]


def _model(c):
    return LearnedPreconditioner(c["nx"], c["ny"], default_kappa(2 * math.pi / c.get("wave", 0.5), c.get("dz", 1.0), 5e-4),
                                 seed=0)


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = _inputs(c, seed)
    s["case"] = c
    if kind in ("cn2d", "pit"):
        e = s["engine"] = CN2D(c["n"], c["nz"], _k(c), 1.0, c["dz"], c["bc"])
        if kind == "pit":
            s["pit"] = PiT2D(e, rtol=1e-6)
        else:
            s["factors"] = e.new_factor_buffer()
            if c["full"]:
                s["store"] = e.new_store(c["probes"])
            s["exit"] = torch.empty((c["probes"], c["n"]), dtype=C64, device="cuda")
    elif kind in ("cn2d_grad", "cn2d_autograd"):
        geo = SimulationGeometry.grid_2d(c["n"], c["nz"], c["wave"], c["probes"], 1, dz=c["dz"])
        s["gradient"] = PWEGradient2D(geo, c["bc"], checkpoint="sqrt" if c["checkpoint"] == "sqrt" else None)
        if kind == "cn2d_autograd":
            s["field"].requires_grad_(True)
    elif kind == "cn3d":
        e = s["engine"] = CN3D(c["nx"], c["ny"], c["nz"], _k(c), 1.0, 1.0, c["dz"], c["bc"])
        s["store"] = e.new_store(c["probes"])
        s["exit"] = torch.empty((c["probes"], e.N), dtype=C64, device="cuda")
    elif kind == "cn3d_grad":
        geo = SimulationGeometry(dimension=3, nx=c["nx"], ny=c["ny"], nz=c["nz"], dx=1.0, dy=1.0, dz=c["dz"], k=_k(c),
                                 num_probes=c["probes"])
        s["gradient"] = PWEGradient3D(geo, c["bc"], precond="learned" if c["learned"] else True,
                                      model=_model(c) if c["learned"] else None)
    elif kind == "ms2d":
        s["engine"] = MS2D(c["n"], c["nz"], _k(c), 1.0, c["dz"])
        s["field"].requires_grad_(True)
    elif kind == "ms3d":
        s["engine"] = MS3D(c["nx"], c["ny"], c["nz"], _k(c), 1.0, 1.0, c["dz"])
        s["field"].requires_grad_(True)
    else:
        s["model"] = _model(c)
    return s


# ------------------------------------------------------------------ the calls
def _single(loss):
    """A loss carries the accuracy of the complex64 exit waves it is computed from."""
    return torch.tensor(loss, dtype=torch.float32)


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "cn2d":
        e = s["engine"]
        fs = e.factor(s["field"], c["mode"], is_delta=c["single"], out=s["factors"])
        start = {"src_exit": s["probes"]} if c["mode"] == "adjoint_exact" else {"probes": s["probes"]}
        e.march(fs, c["probes"], u_store=s.get("store"), exit_out=s["exit"], **start)
        out = {"exit": s["exit"]}
        if c["full"]:
            # the exact adjoint leaves the entrance plane of its store unwritten
            out["field"] = e.unchunk(s["store"]) if c["mode"] != "adjoint_exact" else None
        if heads.fft_plannable(c["n"]):
            out["far"] = heads.farfield_intensity(s["exit"])
        return out
    if kind == "cn2d_grad":
        loss, grad = s["gradient"].loss_and_grad(s["field"], s["probes"], s["amplitude"])
        return {"loss": _single(loss), "gradient": grad}
    if kind == "cn2d_autograd":
        exit_waves = PWEFunction.apply(s["field"], s["probes"], s["gradient"], True)
        (grad,) = torch.autograd.grad(exit_waves, s["field"], s["upstream"])
        return {"exit": exit_waves.detach(), "gradient": grad}
    if kind == "cn3d":
        e = s["engine"]
        e.march(s["field"], c["probes"], c["mode"], probes=s["probes"], u_store=s["store"], exit_out=s["exit"])
        return {"exit": s["exit"], "field": s["store"]}
    if kind == "cn3d_grad":
        loss, grad = s["gradient"].loss_and_grad(s["field"], s["probes"], s["amplitude"])
        return {"loss": _single(loss), "gradient": grad}
    if kind in ("ms2d", "ms3d"):
        function = MSFunction if kind == "ms2d" else MS3DFunction
        exit_waves = function.apply(s["field"], s["probes"], s["engine"])
        (grad,) = torch.autograd.grad(exit_waves, s["field"], s["upstream"])
        # complex64 arithmetic in a complex128 field's gradient
        return {"exit": exit_waves.detach(), "gradient": grad.to(C64)}
    if kind == "pit":
        return {"field": s["pit"].solve(s["field"], probes=s["probes"])}
    loss, gw, gb = s["model"].loss_and_grads(s["diag"], s["z"], s["target"], s["scale"], c["probes"])
    return {"loss": loss, "weights": gw, "biases": gb}


# ------------------------------------------------------------------ work
def work(case):
    """Inputs read once and outputs written once; per row and step about 40 operations for the
    right-hand side and the direct solve of a tridiagonal slice (2D), a 5-point right-hand side and one
    spectral solve (3D), two FFTs and two products (multislice), doubled for a gradient."""
    c, kind = case, case["kind"]
    if kind == "cnn":
        px = c["nx"] * c["ny"] * c["batch"]
        macs = px * 9 * (16 * 32 + 3 * 32 * 32)
        return {"bytes": px * 8 * (1 + 2 * c["probes"]) + 9 * 3584 * 4 * 2, "flops": 6 * macs + px * c["probes"] * 13 * 16}
    P, nz = c["probes"], c["nz"]
    N = c["n"] if "n" in c else c["nx"] * c["ny"]
    fb = 8 if kind == "cn2d_autograd" or c.get("single") else 16
    rows = P * N * (nz - 1)
    by = fb * N * nz + 8 * P * N
    if kind in ("cn2d", "cn3d"):
        by += 8 * P * N + (8 * P * N * nz if kind == "cn3d" or c["full"] else 0)
        return {"bytes": by, "flops": rows * (40 if kind == "cn2d" else 40 + 10 * math.log2(N))}
    if kind == "pit":
        return {"bytes": by + 8 * rows, "flops": rows * 40}
    by += 8 * P * N * (2 if "autograd" in kind or "ms" in kind else 1) + 8 * N * nz
    per = {"cn2d_grad": 40, "cn2d_autograd": 40}.get(kind) or 10 * math.log2(N) + (40 if kind == "cn3d_grad" else 12)
    return {"bytes": by, "flops": rows * (2 * per + 10)}


# ------------------------------------------------------------------ complex128 results
class _Slices:
    """The Crank-Nicolson slices of a case in complex128: K's diagonals for one or two transverse axes
    and the object diagonals c_s.  Solves are Jacobi iterations to round-off (the couplings are small)."""

    def __init__(self, c, dn):
        k, dz = _k(c), c["dz"]
        mu = 1j / (2 * k) * 0.5 * dz
        beta = mu * 2j * k
        self.dims = (c["n"],) if "n" in c else (c["ny"], c["nx"])
        bc, axes = c["bc"], len(self.dims)
        N = math.prod(self.dims)
        one = torch.ones(self.dims, dtype=C128, device="cuda")
        center = -2 * mu * axes * one
        self.off = []
        edge2 = 0.0
        for a, m in enumerate(self.dims):
            lo, hi = mu * one, mu * one
            i = torch.arange(m, device="cuda").reshape([-1 if j == a else 1 for j in range(axes)]).expand(self.dims)
            first, last = i == 0, i == m - 1
            lo, hi = torch.where(first, 0, lo), torch.where(last, 0, hi)
            if bc == "dirichlet":
                hi, lo = torch.where(first, 0, hi), torch.where(last, 0, lo)
            else:
                g = (-1 / (2j * k)) / dz**2 if bc == "impedance2" else 0.0
                hi, lo = torch.where(first, 2 * mu - g, hi), torch.where(last, 2 * mu - g, lo)
                if bc != "neumann":
                    center = center + torch.where(first | last, beta + g, 0.0)
            self.off.append([lo, hi, first | last])
        if bc == "dirichlet":
            # 1D: boundary rows are zero; 2D: the fast axis' edges lose their diagonal and its couplings, the
            # slow axis' edges lose the whole row
            center = torch.where(self.off[-1][2], edge2, center)
            if axes == 2:
                rim = self.off[0][2]
                center = torch.where(rim, 0, center)
                for o in self.off:
                    o[0], o[1] = torch.where(rim, 0, o[0]), torch.where(rim, 0, o[1])
        self.center = center.reshape(N)
        self.off = [[v.reshape(N) for v in o[:2]] for o in self.off]
        coef = -1j * k * dn  # (N, nz), the linearised object term
        self.cs = (dz / 4 * (coef[:, :-1] + coef[:, 1:])).T.contiguous()  # (L, N)
        self.steps = [math.prod(self.dims[a + 1:]) for a in range(axes)]

    def off_apply(self, u, herm):
        out = torch.zeros_like(u)
        for (lo, hi), st in zip(self.off, self.steps):
            if herm:  # (K^H u)_i = conj(hi_{i-st}) u_{i-st} + conj(lo_{i+st}) u_{i+st}
                out[:, st:] += (hi.conj() * u)[:, :-st]
                out[:, :-st] += (lo.conj() * u)[:, st:]
            else:
                out[:, st:] += lo[st:] * u[:, :-st]
                out[:, :-st] += hi[:-st] * u[:, st:]
        return out

    def diag(self, s, herm=False):
        d = self.center + self.cs[s - 1]
        return d.conj() if herm else d

    def apply_p(self, s, u, herm=False):
        return self.diag(s, herm) * u + self.off_apply(u, herm)

    def solve(self, s, b, herm=False):
        """(I - P_s) x = b."""
        inv = 1 / (1 - self.diag(s, herm))
        x = inv * b
        for it in range(200):
            y = inv * (b + self.off_apply(x, herm))
            done = it % 4 == 3 and float((y - x).abs().max()) <= 1e-15 * float(y.abs().max())
            x = y
            if done:
                break
        return x

    def forward(self, u, keep=None):
        for s in range(1, self.cs.shape[0] + 1):
            u = self.solve(s, u + self.apply_p(s, u))
            if keep is not None:
                keep.append(u)
        return u

    def adjoint_gradient(self, src, states):
        """Sum over probes of lambda_s conj(u_s + u_{s-1}) for every slice, (L, N); states u_0 .. u_L."""
        L = self.cs.shape[0]
        acc = torch.empty_like(self.cs)
        b = src
        for s in range(L, 0, -1):
            lam = self.solve(s, b, True)
            acc[s - 1] = (lam * (states[s] + states[s - 1]).conj()).sum(0)
            b = lam + self.apply_p(s, lam, True)
        return acc


def _to_nodes(acc, factor):
    g = torch.zeros((acc.shape[1], acc.shape[0] + 1), dtype=C128, device="cuda")
    g[:, :-1] += acc.T
    g[:, 1:] += acc.T
    return np.conj(factor) * g


def exact(case, seed):
    c, kind = case, case["kind"]
    s = _inputs(c, seed)
    if kind == "cnn":
        return _exact_cnn(c, s)
    u0 = s["probes"].to(C128)
    if kind in ("ms2d", "ms3d"):
        return _exact_multislice(c, s, u0)
    dn = s["field"].to(C128) if kind == "cn2d_autograd" or c.get("single") else s["field"] - 1
    op = _Slices(c, dn)
    L = op.cs.shape[0]
    if kind == "pit":
        # the space-time system takes the probe through B alone
        u = op.solve(1, u0 + op.center * u0 + op.off_apply(u0, False))
        out = [u]
        for t in range(2, L + 1):
            out.append(op.solve(t, out[-1] + op.apply_p(t, out[-1])))
        return {"field": torch.stack(out, 1)}
    if kind in ("cn2d", "cn3d"):
        keep = [u0]
        if c["mode"] == "forward":
            last = op.forward(u0, keep)
        elif c["mode"] == "adjoint":  # the reference's adjoint: conjugate-transposed slices from the last down
            for t in range(L, 0, -1):
                keep.append(op.solve(t, keep[-1] + op.apply_p(t, keep[-1], True), True))
            last = keep[-1]
            keep.reverse()
        else:
            b = u0
            for t in range(L, 0, -1):
                last = op.solve(t, b, True)
                b = last + op.apply_p(t, last, True)
        out = {"exit": last}
        if kind == "cn3d":
            out["field"] = torch.stack(keep, 1)
        else:
            if c["full"]:
                out["field"] = torch.stack(keep, -1) if c["mode"] != "adjoint_exact" else None
            if heads.fft_plannable(c["n"]):
                out["far"] = torch.fft.fft(last, dim=-1).abs() ** 2
        return out
    states = [u0]
    last = op.forward(u0, states)
    factor = c["dz"] / 4 * _k(c) / 1j
    if kind == "cn2d_autograd":
        acc = op.adjoint_gradient(s["upstream"].to(C128), states)
        return {"exit": last, "gradient": _to_nodes(acc, factor)}
    shape, dim = ((-1, c["n"]), (-1,)) if kind == "cn2d_grad" else ((-1, c["nx"], c["ny"]), (-2, -1))
    far = torch.fft.fftn(last.reshape(shape), dim=dim)
    amp, mag = s["amplitude"].reshape(shape), far.abs()
    loss = ((mag - amp) ** 2).sum()
    up = last[0].numel() * torch.fft.ifftn(2 * (mag - amp) * far / mag, dim=dim).reshape(last.shape)
    grad = _to_nodes(op.adjoint_gradient(up, states), factor)
    return {"loss": loss, "gradient": grad if kind == "cn2d_grad" else grad.reshape(c["nx"], c["ny"], c["nz"])}


def _exact_multislice(c, s, u0):
    k, dz, nz = _k(c), c["dz"], c["nz"]
    dims = (c["n"],) if c["kind"] == "ms2d" else (c["nx"], c["ny"])
    dim = tuple(range(-len(dims), 0))
    kt = sum((2 * math.pi * torch.fft.fftfreq(m, dtype=torch.float64, device="cuda").reshape(
        [-1 if j == a else 1 for j in range(len(dims))])) ** 2 for a, m in enumerate(dims))
    H = torch.exp(1j * ((k * k - kt).clamp_min(0).sqrt() - k) * dz)
    T = torch.exp(1j * k * (s["field"] - 1) * dz).T  # (nz, N)
    count, N = u0.shape

    def spread(u, h):
        return torch.fft.ifftn(torch.fft.fftn(u.reshape(count, *dims), dim=dim) * h, dim=dim).reshape(count, N)

    states = [u0]
    for z in range(nz - 1):
        states.append(spread(states[-1] * T[z], H))
    grad = torch.zeros((N, nz), dtype=C128, device="cuda")
    g = s["upstream"].to(C128)
    for z in range(nz - 2, -1, -1):
        g = spread(g, H.conj())
        grad[:, z] = np.conj(1j * k * dz) * (g * (T[z] * states[z]).conj()).sum(0)
        g = g * T[z].conj()
    return {"exit": states[-1], "gradient": grad}


def _exact_cnn(c, s):
    """The network and its gradients in float64 (weights unrounded; the framework computes in bfloat16)."""
    nx, ny, B, per = c["nx"], c["ny"], c["batch"], c["probes"]
    kappa = 1.0 / max(0.5 * 2 * math.pi / 0.5 * 5e-4, 1e-30)
    g = torch.Generator().manual_seed(0)
    ws, bs = [], []
    for i, cin in enumerate((16, 32, 32, 32)):
        std = math.sqrt(2.0 / (9 * cin)) * (1e-2 if i == 3 else 1.0)
        w = (torch.randn((32, cin, 3, 3), generator=g) * std).cuda()
        ws.append(w.double().requires_grad_(True))
        bs.append(torch.zeros(32, dtype=torch.float64, device="cuda", requires_grad=True))
    d = s["diag"].reshape(B, ny, nx).to(C128)
    x = torch.zeros((B, 16, ny, nx), dtype=torch.float64, device="cuda")
    x[:, 0], x[:, 1], x[:, 2] = kappa * d.real, kappa * d.imag, 1.0
    x[:, 3, :, 0], x[:, 4, :, -1], x[:, 5, 0, :], x[:, 6, -1, :] = 1.0, 1.0, 1.0, 1.0
    for i in range(4):
        x = torch.nn.functional.conv2d(x, ws[i], bs[i], padding=1)
        x = torch.relu(x) if i < 3 else x
    z, t = (s[n].to(C128).reshape(B, per, ny, nx) for n in ("z", "target"))
    zp = torch.nn.functional.pad(torch.view_as_real(z), (0, 0, 2, 2, 2, 2))
    zp = torch.view_as_complex(zp.contiguous())
    taps = ((0, 0), (0, -1), (0, 1), (-1, 0), (1, 0), (-1, -1), (-1, 1), (1, -1), (1, 1), (0, -2), (0, 2), (-2, 0), (2, 0))
    y = z
    for j, (dy, dx) in enumerate(taps):
        f = torch.complex(x[:, 2 * j], x[:, 2 * j + 1]) / kappa
        y = y + f[:, None] * zp[:, :, 2 + dy:2 + dy + ny, 2 + dx:2 + dx + nx]
    loss = (s["scale"].double().reshape(B, per, 1, 1) * (y - t).abs() ** 2).sum()
    grads = torch.autograd.grad(loss, ws + bs)
    return {"loss": loss.detach(), "weights": list(grads[:4]), "biases": list(grads[4:])}
