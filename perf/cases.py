"""What a user of this library has it do, as cases that can be timed and compared.

The path in earnest is the device-resident RK3 step (one large tank, uneven
and small tanks, the periodic box, a batch of uneven boxes, the step on host
buffers), the gradient of a tank objective (forward and reverse sweep), and
the operators called on their own: the compact derivatives on device tensors,
the flux divergence on host arrays (the reference's call), the level-set
reinitialisation and the compact filter.  Everything is FP64.

Sizes: the 256^3 tank, the 64^3 Taylor-Green box and the ensemble of grids of
32..160 cells a side are this repository's own configurations; the others are
uneven and small grids of the same workloads.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from emix_gb300 import fields as F
from emix_gb300 import ops


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the tank at the resolution it is run at: one step of a long run
        {"name": "tank_256", "kind": "tank", "nx": 256, "ny": 256, "nz": 256, "steps": 1},
        # a grid fitted to a tank's proportions, no power of two, odd extents
        {"name": "tank_97x121x75", "kind": "tank", "nx": 97, "ny": 121, "nz": 75, "steps": 2},
        # a coarse tank for a quick look at parameters: launches and latency count
        {"name": "tank_40", "kind": "tank", "nx": 40, "ny": 40, "nz": 40, "steps": 4},
        # the 64^3 periodic box with the cyclic scheme
        {"name": "box_64", "kind": "box", "nx": 64, "ny": 64, "nz": 64, "steps": 2},
        # a host program that keeps its fields in its own (page-locked) memory
        {"name": "host_step_160x160x128", "kind": "host", "nx": 160, "ny": 160, "nz": 128, "steps": 1},
        # independent boxes of uneven size advanced together
        {"name": "ensemble_12", "kind": "ensemble", "grids": 12, "draw": 7, "steps": 1},
        # sensitivities of a tank objective: forward and reverse sweep, tapes kept
        {"name": "gradient_96", "kind": "gradient", "nx": 96, "ny": 96, "nz": 96, "steps": 3, "every": 0},
        # velocity and temperature gradients of a field already on the device
        {"name": "deriv_192x160x128", "kind": "deriv", "nx": 192, "ny": 160, "nz": 128, "scheme": "C"},
        # the same on the smallest grids of the tests: the call itself
        {"name": "deriv_24x20x28", "kind": "deriv", "nx": 24, "ny": 20, "nz": 28, "scheme": "B"},
        # the reference's divergence call: host arrays in, host arrays out
        {"name": "divergence_host_96x80x64", "kind": "divergence", "nx": 96, "ny": 80, "nz": 64, "scheme": "C"},
        # reinitialisation of a level set after a few steps
        {"name": "reinit_130x118x106", "kind": "reinit", "nx": 130, "ny": 118, "nz": 106, "iters": 10},
        # the compact filter on the five conserved fields
        {"name": "filter_160x144x128", "kind": "filter", "nx": 160, "ny": 144, "nz": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tank", "tank", "box", "host", "ensemble", "gradient", "deriv", "deriv", "divergence",
                       "reinit", "filter"])
    big = {"tank": 256, "box": 160, "host": 160, "gradient": 104, "deriv": 208, "divergence": 96, "reinit": 130,
           "filter": 160}
    if kind == "ensemble":
        c = {"kind": kind, "grids": rng.randint(3, 12), "draw": rng.randint(1, 10 ** 6), "steps": 1}
        while sum(x * y * z for x, y, z in _ensemble_shapes(c)) > 256 ** 3:
            c["grids"] -= 1
        return c
    lo = 20 if kind in ("deriv", "divergence", "filter", "reinit") else 28
    c = {"kind": kind}
    for a in ("nx", "ny", "nz"):
        c[a] = _log_int(rng, lo, big[kind])
    if kind in ("tank", "box"):
        c["steps"] = rng.choice([1, 1, 2]) if c["nx"] * c["ny"] * c["nz"] < 2 ** 23 else 1
    if kind == "host":
        c["steps"] = 1
    if kind == "gradient":
        c["steps"], c["every"] = rng.choice([2, 3]), rng.choice([0, 0, 1])
    if kind in ("deriv", "divergence"):
        c["scheme"] = rng.choice(["A", "B", "C", "cyclic"])
    if kind == "reinit":
        c["iters"] = 10
    return c


SCHEMES = {"A": F.SCHEME_A, "B": F.SCHEME_B, "C": F.SCHEME_C, "cyclic": F.SCHEME_BPER}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _static(nx, ny, nz, length, origin, periodic):
    """The grid, its metrics and a mask of ones: what a program sets once."""
    g = F.Grid(nx, ny, nz, length, origin, periodic)
    return g, g.jbn(), np.ones(g.shape)


def _axes(g):
    return [torch.from_numpy(g.coords1d(a)).cuda() for a in range(3)]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _modes(g, seed, count=24, kmax=6):
    """Smooth random fields: `count` Fourier modes of up to `kmax` waves over the box, three components, RMS 1."""
    gen = _gen(seed)
    x, y, z = _axes(g)
    k = torch.randint(-kmax, kmax + 1, (3, count), generator=gen, device="cuda").double() * (2 * math.pi)
    ph = torch.rand(count, generator=gen, device="cuda", dtype=torch.float64) * (2 * math.pi)
    amp = torch.randn(3, count, generator=gen, device="cuda", dtype=torch.float64)
    e = [torch.exp(1j * k[a][:, None] * ((c - g.origin[a]) / g.length[a])[None, :]) for a, c in enumerate((x, y, z))]
    zy = (e[2][:, :, None] * e[1][:, None, :] * torch.exp(1j * ph)[:, None, None]).reshape(count, -1).T
    out = torch.stack([((zy * amp[c]) @ e[0]).imag.reshape(g.shape) for c in range(3)])
    return out / out.square().sum(0).mean().sqrt()


def _dt(g, u, mach, cfl):
    cs, most = math.sqrt(1.0 / mach), 0.0
    for a in range(3):
        ua = u[a].abs()
        most = max(most, float(((ua + torch.sqrt(cs * cs + ua * ua)) / (g.length[a] * g.h(a))).max()))
    return cfl / most


def _conserved(p, u, temp, mach):
    r = 1.0 + mach * mach * p
    return torch.stack([r, u[0] * r, u[1] * r, u[2] * r, temp])


def _tank(c, seed, cfl=0.3, mach=0.1):
    """Solid-body rotation with 10% of random modes, a free surface at 0.8 H, a rotating impeller."""
    g, jbn, mask = _static(c["nx"], c["ny"], c["nz"], (2.0, 2.0, 2.0), (-1.0, -1.0, 0.0), (False,) * 3)
    x, y, z = _axes(g)
    omega = 0.8 + 0.4 * float(torch.rand(1, generator=_gen(seed + 17), device="cuda"))
    u = 0.1 * omega * _modes(g, seed)
    u[0] -= omega * y[None, :, None]
    u[1] += omega * x[None, None, :]
    r2 = (x * x)[None, None, :] + (y * y)[None, :, None] + 0 * z[:, None, None]
    um = _conserved(0.5 * omega * omega * r2, u, torch.ones_like(r2), mach)
    phi = (z - 1.6)[:, None, None] + 0 * r2
    w = F.Workload(g, (F.SCHEME_B,) * 3, um.cpu().numpy(), phi.cpu().numpy(), jbn, mask, mach=mach)
    w.dt = _dt(g, u, mach, cfl)
    w.impeller = F.tank_impeller(g, 1.0, 2.0, omega)
    return w, um, phi


def _box(nx, ny, nz, seed, mach=0.1):
    """Taylor-Green flow in a periodic box of side 2 pi with noise of 1e-3, a sphere as the level set."""
    side = 2 * math.pi
    g, jbn, mask = _static(nx, ny, nz, (side,) * 3, (0.0,) * 3, (True,) * 3)
    x, y, z = _axes(g)
    x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
    omega = 0.5 + 1.5 * float(torch.rand(1, generator=_gen(seed + 17), device="cuda"))
    noise = torch.rand((3,) + g.shape, generator=_gen(seed), device="cuda", dtype=torch.float64) * 2 - 1
    one = torch.ones_like(noise[0])
    u = omega * (torch.stack([torch.sin(x) * torch.cos(y) * torch.cos(z) * one,
                              -torch.cos(x) * torch.sin(y) * torch.cos(z) * one, 0 * one]) + 1e-3 * noise)
    p = omega * omega * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0) / 16.0
    um = _conserved(p, u, 1.0 + 0.1 * torch.sin(x) * torch.sin(y) * torch.sin(z) * one, mach)
    m = side / 2
    phi = torch.sqrt((x - m) ** 2 + (y - m) ** 2 + (z - m) ** 2) - 0.25 * side
    w = F.Workload(g, (F.SCHEME_BPER,) * 3, um.cpu().numpy(), phi.cpu().numpy(), jbn, mask, mach=mach)
    w.dt = _dt(g, u, mach, 0.3)
    return w, um, phi


class _View:
    """A device buffer of the library as torch sees one; the tensor made of it keeps the buffer's owner."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f8", "version": 3}


def _view(ptr, shape, owner):
    t = torch.as_tensor(_View(ptr, shape, owner), device="cuda")
    t.owner = owner
    return t


def _spectrum(shape, count, seed):
    """`count` smooth fields of order one with noise of 1e-2, as gradients and divergences are taken of."""
    g = F.Grid(shape[2], shape[1], shape[0])
    a = torch.cat([_modes(g, seed + 31 * k, 12, 4) for k in range((count + 2) // 3)])[:count]
    return (a + 0.01 * torch.randn(a.shape, generator=_gen(seed + 5), device="cuda", dtype=torch.float64)).contiguous()


def _ensemble_shapes(c):
    return F.ensemble_shapes(c["grids"], c["draw"])


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"kind": kind, "case": c}
    if kind in ("tank", "box"):
        if kind == "tank":
            w, um, phi = _tank(c, seed)
            ctx = ops.Context(w, bc_walls=1)
        else:
            w, um, phi = _box(c["nx"], c["ny"], c["nz"], seed)
            ctx = ops.Context(w)
        # torch works on the context's stream, so that its copies and the steps follow one another
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        pu, pp = ctx.state_ptrs()
        s |= {"ctx": ctx, "stream": stream, "um0": um, "phi0": phi, "um": _view(pu, tuple(um.shape), ctx),
              "phi": _view(pp, tuple(phi.shape), ctx)}
    elif kind == "host":
        w, um, phi = _tank(c, seed, cfl=0.1)
        ctx = ops.Context(w, bc_walls=1)
        hum, hphi = um.cpu().pin_memory(), phi.cpu().pin_memory()
        s |= {"ctx": ctx, "um": hum, "phi": hphi, "keep": (hum.numpy(), hphi.numpy())}
    elif kind == "ensemble":
        made = [_box(*shape, seed + 101 * k) for k, shape in enumerate(_ensemble_shapes(c))]
        b = ops.Batch([m[0] for m in made])
        stream = torch.cuda.Stream()
        b.set_stream(stream.cuda_stream)
        state = []
        for h, (w, um, phi) in zip(b.ctx, made):
            pu, pp = ops.C.c_void_p(), ops.C.c_void_p()
            ops.check(b.lib.emix_ctx_state(h, ops.C.byref(pu), ops.C.byref(pp)), "emix_ctx_state")
            state.append((_view(pu.value, tuple(um.shape), b), _view(pp.value, tuple(phi.shape), b), um, phi))
        s |= {"batch": b, "stream": stream, "state": state}
    elif kind == "gradient":
        w, um, phi = _tank(c, seed)
        grad = ops.TankGradient(w, c["steps"], every=c["every"], bc_walls=1)
        s |= {"grad": grad, "omega": w.impeller.omega, "cs": w.cs}
    elif kind == "deriv":
        a = _spectrum((c["nz"], c["ny"], c["nx"]), 4, seed)
        s |= {"vel": a[:3].contiguous(), "temp": a[3].contiguous(), "h": _spacings(c)}
    elif kind == "divergence":
        a = _spectrum((c["nz"], c["ny"], c["nx"]), 6, seed)
        s |= {"flux": [np.ascontiguousarray(q) for q in a.cpu().numpy()], "h": _spacings(c),
              "jbn": F.Grid(c["nx"], c["ny"], c["nz"], (1.3, 0.9, 1.1)).jbn()}
    elif kind == "reinit":
        n = (c["nz"] + 10, c["ny"] + 10, c["nx"] + 10)
        g = F.Grid(n[2], n[1], n[0], (1.0, 1.0, 1.0))
        x, y, z = _axes(g)
        d = torch.sqrt((x - 0.5)[None, None, :] ** 2 + (y - 0.45)[None, :, None] ** 2 + (z - 0.55)[:, None, None] ** 2) - 0.3
        phi0 = d * (1.0 + 0.3 * _modes(g, seed, 8, 2)[0])
        dm = min(g.h(a) for a in range(3))
        s |= {"phi0": phi0, "phi": torch.empty_like(phi0), "jbn": torch.from_numpy(g.jbn()).cuda(),
              "dmins": torch.full(n, dm, dtype=torch.float64, device="cuda"), "delta": tuple(g.h(a) for a in range(3)),
              "dm": dm}
    elif kind == "filter":
        g = F.Grid(c["nx"], c["ny"], c["nz"], (2.0, 2.0, 2.0))
        s |= {"um0": _spectrum(g.shape, 5, seed), "jbn": torch.from_numpy(g.jbn()).cuda()}
        s["um"] = torch.empty_like(s["um0"])
    return s


def _spacings(c):
    per = c["scheme"] == "cyclic"
    return tuple(1.0 / n if per else 1.0 / (n - 1) for n in (c["nx"], c["ny"], c["nz"]))


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(s):
    kind, c = s["kind"], s["case"]
    if kind in ("tank", "box"):
        # a run started from a saved state
        with torch.cuda.stream(s["stream"]):
            s["um"].copy_(s["um0"])
            s["phi"].copy_(s["phi0"])
        s["ctx"].step(c["steps"], use_graph=True)
        return {"um": s["um"], "phi": s["phi"]}
    if kind == "host":
        # the program's own buffers, advanced in place call after call
        s["ctx"].step_host(s["keep"][0], s["keep"][1], c["steps"])
        return {"um": s["um"], "phi": s["phi"]}
    if kind == "ensemble":
        with torch.cuda.stream(s["stream"]):
            for um, phi, um0, phi0 in s["state"]:
                um.copy_(um0)
                phi.copy_(phi0)
        s["batch"].step(c["steps"], use_graph=True)
        return [[um, phi] for um, phi, _, _ in s["state"]]
    if kind == "gradient":
        J = s["grad"].run(s["omega"], s["cs"])
        dJ = s["grad"].adj.backward()
        lum, lphi = s["grad"].adj.state_gradient()
        return {"J": J, "dJ": list(dJ), "lum": lum, "lphi": lphi}
    if kind == "deriv":
        return list(ops.cudaDeriv_dev(s["vel"], s["temp"], s["h"], SCHEMES[c["scheme"]]))
    if kind == "divergence":
        return list(ops.cuDivergence(*s["flux"], s["jbn"], s["h"], SCHEMES[c["scheme"]]))
    if kind == "reinit":
        s["phi"].copy_(s["phi0"])
        ops.reinit_dev(s["phi"], s["jbn"], s["dmins"], s["delta"], 5, s["dm"], iters=c["iters"])
        return s["phi"]
    if kind == "filter":
        s["um"].copy_(s["um0"])
        ops.filtrado_dev(s["um"], s["jbn"], 0.45)
        return s["um"]
    raise ValueError(kind)


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind == "ensemble":
        n = sum(x * y * z for x, y, z in _ensemble_shapes(c))
    else:
        n = c["nx"] * c["ny"] * c["nz"]
    if kind in ("tank", "box", "host", "ensemble"):
        # state in and out (6 + 6), metrics, mask and filter width (13); about
        # 1050 FP64 operations per cell and step, a third of them fused
        return {"bytes": 8.0 * 25 * n * c["steps"], "flops": 1400.0 * n * c["steps"]}
    if kind == "gradient":
        return {"bytes": 8.0 * (25 + 12) * n * c["steps"], "flops": 4000.0 * n * c["steps"]}
    if kind == "deriv":
        return {"bytes": 8.0 * 16 * n, "flops": 8.0 * 12 * n}
    if kind == "divergence":
        return {"bytes": 8.0 * (6 + 4 + 2) * n, "flops": 8.0 * 6 * n + 16.0 * n}
    if kind == "reinit":
        m = (c["nx"] + 10) * (c["ny"] + 10) * (c["nz"] + 10)
        return {"bytes": 8.0 * 7 * m, "flops": 3.0 * c["iters"] * 180 * m}
    return {"bytes": 8.0 * 12 * n, "flops": 5.0 * 3 * 18 * n}


# --------------------------------------------------------------------------
# the operators in 64 bits, by dense matrices
# --------------------------------------------------------------------------
def _dense(scheme, n, h):
    """The compact first derivative A f' = B f / h as a dense matrix A^-1 B / h."""
    A, B = torch.eye(n, dtype=torch.float64), torch.zeros(n, n, dtype=torch.float64)
    al, a, b = (0.25, 0.75, 0.0) if scheme == "A" else (1.0 / 3.0, 7.0 / 9.0, 1.0 / 36.0)
    for i in range(n):
        for d, v in ((1, a), (-1, -a), (2, b), (-2, -b)):
            B[i, (i + d) % n] += v
        A[i, (i + 1) % n] += al
        A[i, (i - 1) % n] += al
    if scheme != "cyclic":
        first = (2.0, [-2.5, 2.0, 0.5, 0.0]) if scheme == "B" else (3.0, [-17.0 / 6.0, 1.5, 1.5, -1.0 / 6.0])
        for i, sign in ((0, 1.0), (1, 1.0), (n - 2, -1.0), (n - 1, -1.0)):
            A[i], B[i], step = 0.0, 0.0, int(sign)
            A[i, i] = 1.0
            if i in (0, n - 1):
                A[i, i + step] = first[0]
                for k, v in enumerate(first[1]):
                    B[i, i + step * k] = sign * v
            else:
                A[i, i - 1] = A[i, i + 1] = 0.25
                B[i, i + 1], B[i, i - 1] = 0.75, -0.75
    return torch.linalg.solve(A, B / h).cuda()


def _along(D, f, axis):
    return torch.movedim(torch.movedim(f, -1 - axis, -1) @ D.T, -1, -1 - axis)


def exact(case, seed):
    """The derivatives and the divergence by dense matrices; whole steps, the
    gradient through them, the reinitialisation and the filter have no short
    plain form."""
    if case["kind"] not in ("deriv", "divergence"):
        return None
    c, s = case, prepare(case, seed)
    D = [_dense(c["scheme"], n, h) for n, h in zip((c["nx"], c["ny"], c["nz"]), s["h"])]
    if c["kind"] == "deriv":
        dvel = torch.cat([_along(D[a], s["vel"], a) for a in range(3)])
        return [dvel, torch.stack([_along(D[a], s["temp"], a) for a in range(3)])]
    j = torch.from_numpy(s["jbn"]).cuda()
    f = [torch.from_numpy(q).cuda() for q in s["flux"]]
    out = []
    for part in (f[:3], f[3:]):
        out.append((j[10] * sum(_along(D[a], j[9] * (j[4 * a] * part[a]), a) for a in range(3))).cpu().numpy())
    return out
