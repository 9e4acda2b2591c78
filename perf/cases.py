"""The workloads whose speed and accuracy are measured, each through the
public entry points a user's program calls:

  kick      ``SpaceChargeCalc2p5D.trackBunch(bunch, length)``: one 2.5D
            space-charge kick outside a lattice program
  rb        ``SpaceChargeCalc2p5Drb.trackBunch(bunch, length, pipe_radius)``
  boundary  ``SpaceChargeCalc2p5D.trackBunch(bunch, length, boundary)`` with
            a circular conducting boundary
  fodo      one ``TEAPOT_Lattice.trackBunch(bunch)`` through a FODO line with
            four 2.5D kicks per cell (plain FP64, FP32 field form, or the
            learned closure over the FP32 form)
  ring      the same call through ring cells with quadrupoles, sextupoles and
            sector bends
  batch     ``BunchBatch.trackTurns(1)``: many bunches, each with its own
            lattice and grid
  diag      ``BunchTwissAnalysis.computeBunchMoments`` (with analyzeBunch)
  train     ``DeviceDenoiser.gradients``: forward, loss and backward of the
            denoising network on a batch of density images

``listed()`` gives the fixed cases, ``draw(rng)`` more of the same ranges;
``prepare`` makes the bunch, calculator and lattice a program holds, ``run``
is one pass, and ``exact`` the same result from plain torch in 64 bits.
"""
import contextlib
import io
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "py-orbit_gb300")

KIN_ENERGY = 1.0  # GeV protons
MASS = 0.938272013
R_CLASSICAL = 1.534698e-18
PROTONS = 1e14


def _package():
    if _PKG not in sys.path:
        sys.path.insert(0, _PKG)


def listed():
    return [
        # the smallest call: a quick check of a beam, where launches and the wait count
        {"name": "kick_small", "kind": "kick", "n": 10_000, "nx": 64, "ny": 64, "nz": 1, "form": "plain",
         "msize": False},
        # an odd bunch on a grid that is no power of two, every particle with its own macrosize
        {"name": "kick_ragged", "kind": "kick", "n": 333_333, "nx": 96, "ny": 80, "nz": 48, "form": "plain",
         "msize": True},
        # a short line with few particles: one point of a matching loop
        {"name": "fodo_small", "kind": "fodo", "n": 20_011, "nx": 64, "ny": 64, "nz": 32, "cells": 4,
         "kq": 0.5, "form": "plain"},
        # the benchmark line at its own size, a quarter of a turn (40 kicks)
        {"name": "fodo_1m", "kind": "fodo", "n": 1_000_000, "nx": 128, "ny": 128, "nz": 64, "cells": 10,
         "kq": 0.5, "form": "plain"},
        # the same line with the field in FP32
        {"name": "fodo_fp32", "kind": "fodo", "n": 1_000_000, "nx": 128, "ny": 128, "nz": 64, "cells": 4,
         "kq": 0.5, "form": "fp32"},
        # few particles and the denoising network inside every kick
        {"name": "fodo_learned", "kind": "fodo", "n": 100_000, "nx": 128, "ny": 128, "nz": 64, "cells": 4,
         "kq": 0.5, "form": "learned"},
        # the largest bunch and grid: a quarter of the ring
        {"name": "ring_16m", "kind": "ring", "n": 16_000_000, "nx": 256, "ny": 256, "nz": 128, "cells": 8},
        # an intensity and strength scan of uneven bunches on three grid sizes
        {"name": "batch_scan", "kind": "batch", "members": 12, "n_max": 1_000_000, "cells": 4},
        # the kick with the longitudinal part and a pipe
        {"name": "rb_2m", "kind": "rb", "n": 2_000_000, "nx": 128, "ny": 128, "nz": 64},
        # the kick inside a conducting pipe
        {"name": "boundary_1m", "kind": "boundary", "n": 1_000_000, "nx": 128, "ny": 128, "nz": 32,
         "points": 128, "modes": 10},
        # moments and emittances of a tracked bunch, read every few turns
        {"name": "diag_4m", "kind": "diag", "n": 4_000_003, "order": 4},
        # one step's gradients of the network's training
        {"name": "train_16", "kind": "train", "batch": 16, "size": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_GRID = (32, 40, 48, 64, 80, 96, 100, 112, 128, 160, 192, 256)


def draw(rng):
    kind = rng.choice(("kick", "kick", "fodo", "fodo", "fodo", "ring", "batch", "rb", "boundary", "diag", "train"))
    if kind in ("kick", "rb", "boundary"):
        msize = kind == "kick" and rng.random() < 0.25
        case = {"kind": kind, "n": _log(rng, 2_000, 300_000 if msize else 4_000_000), "nx": rng.choice(_GRID),
                "ny": rng.choice(_GRID), "nz": _log(rng, 1, 128)}
        if kind == "kick":
            case.update(form="plain" if msize else rng.choice(("plain", "plain", "fp32")), msize=msize)
        if kind == "boundary":
            case.update(points=4 * _log(rng, 16, 64), modes=rng.randint(4, 14))
        if kind == "rb":
            case["nz"] = max(case["nz"], 4)
        return case
    if kind == "fodo":
        form = rng.choice(("plain", "plain", "fp32", "learned"))
        if form == "learned":
            return {"kind": kind, "n": _log(rng, 50_000, 200_000), "nx": 128, "ny": 128, "nz": _log(rng, 16, 64),
                    "cells": rng.randint(2, 4), "kq": round(rng.uniform(0.35, 0.6), 3), "form": form}
        # a space-charge line amplifies a change of rounding from cell to cell,
        # the more so the fewer the particles and the coarser the field
        n = _log(rng, 5_000, 1_500_000)
        cells = rng.randint(2, 4) if form == "fp32" or n < 100_000 else _log(rng, 2, 10)
        nx = rng.choice(_GRID)
        ny = nx if rng.random() < 0.6 else rng.choice(_GRID)
        return {"kind": kind, "n": n, "nx": nx, "ny": ny, "nz": _log(rng, 8, 128),
                "cells": cells, "kq": round(rng.uniform(0.35, 0.6), 3), "form": form}
    if kind == "ring":
        g = rng.choice((128, 192, 256))
        return {"kind": kind, "n": _log(rng, 200_000, 16_000_000), "nx": g, "ny": g, "nz": _log(rng, 32, 128),
                "cells": rng.randint(1, 8)}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(3, 14), "n_max": _log(rng, 100_000, 1_000_000),
                "cells": rng.randint(1, 4)}
    if kind == "diag":
        return {"kind": kind, "n": _log(rng, 20_000, 8_000_000), "order": rng.randint(2, 5)}
    return {"kind": "train", "batch": rng.randint(2, 16), "size": rng.choice((64, 96, 128))}


# ---------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed, k=0):
    return torch.Generator(device=_device()).manual_seed(int(seed) * 1009 + k)


def _normal(n, g):
    return torch.randn(n, generator=g, device=g.device, dtype=torch.float64)


def _uniform(shape, g):
    return torch.rand(shape, generator=g, device=g.device, dtype=torch.float64)


def _waterbag(n, g, rms=4e-3, rmsp=0.8e-3):
    """4D waterbag (a uniform 4D ball), z ~ N(0, 10 m), dE ~ N(0, 1 MeV)."""
    u = torch.stack([_normal(n, g) for _ in range(4)])
    u *= _uniform((n,), g) ** 0.25 / u.norm(dim=0) * math.sqrt(6.0)
    return torch.stack([rms * u[0], rmsp * u[1], rms * u[2], rmsp * u[3], 10.0 * _normal(n, g), 1e-3 * _normal(n, g)])


def _gauss(n, g):
    return torch.stack([4e-3 * _normal(n, g), 0.8e-3 * _normal(n, g), 4e-3 * _normal(n, g), 0.8e-3 * _normal(n, g),
                        10.0 * _normal(n, g), 1e-3 * _normal(n, g)])


def _kv_parabolic(n, g):
    """4D KV (the surface of a 4D ball), parabolic line density over 250 m."""
    u = torch.stack([_normal(n, g) for _ in range(4)])
    u /= u.norm(dim=0)
    w = 2.0 * _uniform((3, n), g) - 1.0
    z = 125.0 * w.median(dim=0).values
    return torch.stack([12e-3 * u[0], 2e-3 * u[1], 12e-3 * u[2], 2e-3 * u[3], z, 1e-3 * _normal(n, g)])


def _beam(case, seed):
    """(coordinates, macrosize, per-particle macrosizes or None)."""
    g, n = _gen(seed), case["n"]
    if case["kind"] == "ring":
        return _kv_parabolic(n, g), PROTONS / n, None
    if case["kind"] == "diag":
        c = _gauss(n, g)
        c[1] -= 0.05 * c[0]
        c[0] += 1e-3 + 0.4 * c[5]
        return c, PROTONS / n, None
    if case["kind"] == "kick" and not case["msize"]:
        c = _gauss(n, g)
        c[4] = 200.0 * _uniform((n,), g) - 100.0
        return c, PROTONS / n, None
    c = _waterbag(n, g)
    m = (0.5 + _uniform((n,), g)) * (PROTONS / n) if case.get("msize") else None
    return c, PROTONS / n, m


_SCAN_GRIDS = ((64, 64, 32), (128, 128, 64), (256, 256, 64))


def _scan(case, seed):
    """[(particles, grid, k1, protons)] of a scan; the sizes belong to the
    case, the strengths and intensities to the seed."""
    out = []
    for k in range(case["members"]):
        n = int(5e4 * (case["n_max"] / 5e4) ** ((k * 7 % case["members"]) / max(1, case["members"] - 1))) + 3 * k
        u = np.random.RandomState((int(seed) * 131 + k) % (1 << 31)).uniform(size=2)
        out.append((n, _SCAN_GRIDS[k % 3], 0.35 + 0.25 * u[0], 1e13 * 10.0 ** u[1]))
    return out


def _images(case, seed):
    """Normalised densities: smooth beams and what 1e5 particles show of them."""
    g, s, nb = _gen(seed), case["size"], case["batch"]
    ax = torch.linspace(-1.0, 1.0, s, device=g.device, dtype=torch.float64)
    a = 0.35 + 0.5 * _uniform((nb, 2), g)
    p = 0.5 + 1.5 * _uniform((nb, 1, 1), g)
    r2 = (ax[None, :, None] / a[:, 0, None, None]) ** 2 + (ax[None, None, :] / a[:, 1, None, None]) ** 2
    t = (1.0 - r2).clamp(min=0.0) ** p
    t = t / t.mean(dim=(1, 2), keepdim=True)
    per = 1e5 / (s * s)
    x = torch.poisson(t * per, generator=g) / per
    return x[:, None].float().contiguous(), t[:, None].float().contiguous()


# ---------------------------------------------------------------------
# the program's objects and one pass
# ---------------------------------------------------------------------
class _Row:
    """A device row of FP64 coordinates by address, for torch.as_tensor."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": "<f8", "data": (int(ptr), False), "version": 3}


def _bunch(coords, macrosize, msize=None):
    """A Bunch on the GPU and its six coordinate rows."""
    from bunch import Bunch
    b = Bunch()
    b.getSyncParticle().kinEnergy(KIN_ENERGY)
    b.macroSize(macrosize)
    b.setCoordinates(coords.cpu().numpy(), copy=False)
    if msize is not None:
        b.addPartAttr("macrosize")
        for i, v in enumerate(msize.cpu().tolist()):
            b.partAttrValue("macrosize", i, 0, v)
    dev = b._device_bunch()
    return b, [torch.as_tensor(_Row(p, coords.shape[1]), device="cuda") for p in dev.device_pointers()]


@contextlib.contextmanager
def _quiet():
    with contextlib.redirect_stdout(io.StringIO()):
        yield


PIPE_RADIUS = 0.05
PIPE = 0.04  # diameter of the circular boundary
KICK_LENGTH = 0.5


def prepare(case, seed):
    _package()
    from orbit_gb300 import denoiser, workloads
    from spacecharge import Boundary2D, SpaceChargeCalc2p5D, SpaceChargeCalc2p5Drb
    kind = case["kind"]
    if kind == "train":
        net = denoiser.default_network(max_batch=case["batch"], size=case["size"])
        net.set_batch_tensor_cores(True)
        x, t = _images(case, seed)
        return {"kind": kind, "net": net, "x": x, "t": t, "y": torch.empty_like(x)}
    if kind == "batch":
        from orbit_gb300.batch import BunchBatch
        members, rows = [], []
        for k, (n, grid, k1, protons) in enumerate(_scan(case, seed)):
            b, r = _bunch(_gauss(n, _gen(seed, 1 + k)), protons / n)
            with _quiet():
                lat = workloads.fodo_lattice(SpaceChargeCalc2p5D(*grid), cells=case["cells"], kq=k1)
            members.append((b, lat))
            rows.append(r)
        return {"kind": kind, "batch": BunchBatch(members), "rows": rows}
    coords, macrosize, msize = _beam(case, seed)
    b, rows = _bunch(coords, macrosize, msize)
    state = {"kind": kind, "bunch": b, "rows": rows}
    if kind == "diag":
        from bunch import BunchTwissAnalysis
        state.update(twiss=BunchTwissAnalysis(), order=case["order"])
    elif kind == "kick":
        state["calc"] = SpaceChargeCalc2p5D(case["nx"], case["ny"], case["nz"], form=case["form"])
    elif kind == "rb":
        state["calc"] = SpaceChargeCalc2p5Drb(case["nx"], case["ny"], case["nz"])
    elif kind == "boundary":
        state["calc"] = SpaceChargeCalc2p5D(case["nx"], case["ny"], case["nz"])
        state["boundary"] = Boundary2D(case["points"], case["modes"], "Circle", PIPE)
    elif kind == "ring":
        with _quiet():
            state["lattice"] = workloads.ring_lattice(SpaceChargeCalc2p5D(case["nx"], case["ny"], case["nz"]),
                                                      cells=case["cells"])
    else:
        calc = SpaceChargeCalc2p5D(case["nx"], case["ny"], case["nz"],
                                   form="plain" if case["form"] == "plain" else "fp32")
        if case["form"] == "learned":
            state["net"] = denoiser.default_network()
            calc.setDenoiser(state["net"])
        with _quiet():
            state["lattice"] = workloads.fodo_lattice(calc, cells=case["cells"], kq=case["kq"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "train":
        loss, grads = state["net"].gradients(state["x"].data_ptr(), state["t"].data_ptr(), state["x"].shape[0],
                                             dev_out=state["y"].data_ptr())
        return {"loss": loss, "grads": grads, "y": state["y"]}
    if kind == "batch":
        state["batch"].trackTurns(1)
        return [r for rows in state["rows"] for r in (rows[0], rows[1], rows[3], rows[4])]
    b = state["bunch"]
    if kind == "diag":
        tw, order = state["twiss"], state["order"]
        tw.computeBunchMoments(b, order)
        return {"avg": np.array([tw.getAverage(i) for i in range(6)]),
                "corr": np.array([[tw.getCorrelation(i, j) for j in range(6)] for i in range(6)]),
                "emit": np.array([tw.getEmittance(i) for i in range(2)]),
                "moments": np.array([[tw.getBunchMoment(i, j) for j in range(order + 1)] for i in range(order + 1)])}
    if kind == "kick":
        state["calc"].trackBunch(b, KICK_LENGTH)
    elif kind == "rb":
        state["calc"].trackBunch(b, KICK_LENGTH, PIPE_RADIUS)
    elif kind == "boundary":
        state["calc"].trackBunch(b, KICK_LENGTH, state["boundary"])
    else:
        state["lattice"].trackBunch(b)
    return state["rows"]


# ---------------------------------------------------------------------
# work
# ---------------------------------------------------------------------
_NET_FLOPS = 1.19e9 / 16384  # one forward of the network, per pixel


def _solve_flops(nx, ny):
    """Forward and backward transforms of the doubled grid and the product."""
    n = 4.0 * nx * ny
    return 2 * 2.5 * n * math.log2(n) + 6 * n / 2


def _line_work(n, nx, ny, nz, kicks, maps):
    """One pass of a line: coordinates in and out once, the kick's, the
    deposit's and the maps' operations of every particle and kick."""
    return {"bytes": 96.0 * n, "flops": kicks * (n * (113.0 + 69.0 + maps) + _solve_flops(nx, ny))}


def work(case):
    kind = case["kind"]
    if kind == "train":
        pix = case["batch"] * case["size"] ** 2
        return {"bytes": 12.0 * pix + 8.0 * 302_561, "flops": 3 * _NET_FLOPS * pix}
    if kind == "batch":
        parts = [_line_work(n, *grid, 4 * case["cells"], 117.0) for n, grid, _, _ in _scan(case, 1)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["n"]
    if kind == "diag":
        cells = (case["order"] + 1) * (case["order"] + 2) / 2
        return {"bytes": 48.0 * n, "flops": n * (27 * 2.0 + cells * 4.0)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind in ("kick", "boundary"):
        return {"bytes": (56.0 + 8.0 * bool(case.get("msize"))) * n, "flops": n * 182.0 + _solve_flops(nx, ny)}
    if kind == "rb":
        return {"bytes": 72.0 * n, "flops": n * 205.0 + _solve_flops(nx, ny)}
    if kind == "ring":
        return _line_work(n, nx, ny, nz, len([1 for o in _ring_ops(case["cells"]) if o[0] == "sc"]), 330.0)
    w = _line_work(n, nx, ny, nz, 4 * case["cells"], 117.0)
    if case["form"] == "learned":
        w["flops"] += 4 * case["cells"] * _NET_FLOPS * nx * ny
    return w


# ---------------------------------------------------------------------
# the same results in 64 bits from plain torch
# ---------------------------------------------------------------------
def _kinematics():
    gamma = (KIN_ENERGY + MASS) / MASS
    beta = math.sqrt(1.0 - 1.0 / gamma ** 2)
    return beta, gamma, math.sqrt(KIN_ENERGY * (KIN_ENERGY + 2.0 * MASS))


def _place_kicks(nodes, sc_min):
    """The op list of nodes [(entrance ops, [(part length, ops)], exit ops)]
    with a kick before every part that starts after more than sc_min of
    path, and one at the start; each kicks for the path to the next."""
    marks, since, walked = [], 0.0, 0.0
    for k, (_, parts, _) in enumerate(nodes):
        for p, (length, _) in enumerate(parts):
            if since > sc_min:
                marks.append(((k, p), walked, since))
                since = 0.0
            since += length
            walked += length
    at = [(0, 0)] + [m[0] for m in marks]
    lengths = [m[2] for m in marks] + [walked - (marks[-1][1] if marks else 0.0)]
    kick = dict(zip(at, lengths))
    ops = []
    for k, (first, parts, last) in enumerate(nodes):
        ops += first
        for p, (_, body) in enumerate(parts):
            if (k, p) in kick:
                ops.append(("sc", kick[k, p]))
            ops += body
        ops += last
    return ops


def _quad(length, kq):
    h = length / 2.0
    return ([("qfringe", kq)], [(h, [("quad1", h, kq)]), (h, [("quad2", h), ("quad2", h), ("quad1", h, kq)])],
            [("qfringe", -kq)])


def _drift(length):
    return ([], [(length, [("drift", length)])], [])


def _sextupole(length, k2):
    h = length / 2.0
    return ([("mfringe", 2, -k2)], [(h, [("drift", h)]), (h, [("multipole", 2, k2 * length), ("drift", h)])],
            [("mfringe", 2, k2)])


def _bend(length, theta):
    h, th = length / 2.0, theta / 2.0
    rho = length / theta
    one = ("bend1", h, th)
    return ([("bfringe", rho)],
            [(h, [one]), (h, [("quad2", h), ("bend3", th), ("bend4", th), ("bend4", th), ("bend3", th), ("quad2", h),
                              one])],
            [("bfringe", -rho)])


def _fodo_ops(cells, kq):
    return _place_kicks([e for _ in range(cells) for e in (_quad(0.5, kq), _drift(2.0), _quad(0.5, -kq), _drift(2.0))],
                        0.3)


def _ring_ops(cells):
    nodes = []
    for c in range(cells):
        nodes += [_quad(0.5, 0.5)] + ([_drift(0.85), _drift(0.85)] if c < 12 else [_drift(1.7)])
        nodes += [_sextupole(0.2, 2.0), _drift(0.5), _bend(2.0, 2.0 * math.pi / 32), _drift(0.5), _quad(0.5, -0.5),
                  _drift(1.7), _sextupole(0.2, -2.0)]
    return _place_kicks(nodes, 1.4)


def _map(op, c):
    """One TEAPOT map on the rows of c."""
    beta, gamma, momentum = _kinematics()
    g2 = 1.0 / gamma ** 2
    x, xp, y, yp, z = (c[k].clone() for k in range(5))
    d = c[5] / (momentum * beta)
    k = 1.0 / (1.0 + d)
    name = op[0]
    if name == "drift":
        c[0] += k * op[1] * xp
        c[2] += k * op[1] * yp
        f = 0.5 * (xp * xp + yp * yp + d * d * g2)
        c[4] -= op[1] * (f * k - d * g2) * k
    elif name == "quad1":
        length, kq = op[1], op[2]
        s = math.sqrt(abs(kq))
        focus = (math.cos(s * length), math.sin(s * length) / s, -math.sin(s * length) * s)
        defoc = (math.cosh(s * length), math.sinh(s * length) / s, math.sinh(s * length) * s)
        hx, hy = (focus, defoc) if kq > 0 else (defoc, focus)
        c[0], c[1] = hx[0] * x + hx[1] * xp, hx[2] * x + hx[0] * xp
        c[2], c[3] = hy[0] * y + hy[1] * yp, hy[2] * y + hy[0] * yp
        c[4] += d * g2 * length
    elif name == "quad2":
        length = op[1]
        c[0] -= k * length * d * xp
        c[2] -= k * length * d * yp
        f = 0.5 * (xp * xp + yp * yp + d * d * g2)
        c[4] -= length * (f * k + d * d * g2) * k
    elif name == "qfringe":
        q = op[1] * k
        a = q / 4.0 * (x * x + y * y)
        b = q / 2.0 * x * y
        det = 1.0 - (q / 4.0 * (x * x - y * y)) ** 2
        c[1] = (xp - a * xp + b * yp) / det
        c[3] = (yp + a * yp - b * xp) / det
        fx = q / 12.0 * x * (x * x + 3.0 * y * y)
        fy = q / 12.0 * y * (y * y + 3.0 * x * x)
        c[0] += fx
        c[2] -= fy
        c[4] += k * (xp * fx - yp * fy)
    elif name == "bend1":
        length, th = op[1], op[2]
        rho, cs, sn = length / th, math.cos(th), math.sin(th)
        c[0] = cs * x + rho * sn * xp + rho * (1.0 - cs) * d
        c[1] = -sn / rho * x + cs * xp + sn * d
        c[2] += length * yp
        c[4] += -sn * x - rho * (1.0 - cs) * xp + (rho * sn - beta * beta * length) * d
    elif name == "bend3":
        th = op[1]
        f = 0.5 * (yp * yp + d * d * g2)
        c[1] -= f * k * th
        c[2] += k * yp * x * th
        c[4] -= th * (f * k - d * g2) * k * x
    elif name == "bend4":
        th = op[1]
        a = 1.0 + 0.5 * k * xp * th
        c[0] = x * a * a
        c[1] = xp / a
        c[4] -= th * 0.5 * (k * xp) ** 2 * c[0]
    elif name == "bfringe":
        h = 1.0 / op[1]
        c[0] += 0.5 * h * k * y * y
        c[3] -= h * k * xp * y
        c[4] += 0.5 * h * k * k * xp * y * y
    elif name == "multipole":
        w = torch.complex(x, y) ** op[1] * (op[2] / math.factorial(op[1]))
        c[1] -= w.real
        c[3] += w.imag
    elif name == "mfringe":
        # generating function with the signed strength kt: with l = pole + 1,
        # A + iB = kt w^(l-1), C + iD = kt w^l (w = x + i y)
        pole, l = op[1], op[1] + 1.0
        kt = op[2] / (4.0 * math.factorial(pole + 2))
        w = torch.complex(x, y)
        wl = w ** pole
        A, B = kt * wl.real, kt * wl.imag
        C, D = A * x - B * y, A * y + B * x
        fx, fy = l * C * x + (l + 2) * D * y, l * C * y - (l + 2) * D * x
        dxfx = l * (l + 1) * (A * x + B * y)
        dyfx = (l + 1) * (l + 2) * A * y - (l + 1) * (l - 2) * B * x
        dxfy = (l + 1) * (l - 2) * A * y - (l + 1) * (l + 2) * B * x
        m11, m12, m21, m22 = 1.0 - dxfx * k, -dxfy * k, -dyfx * k, 1.0 + dxfx * k
        det = m11 * m22 - m12 * m21
        c[1] = (m22 * xp - m12 * yp) / det
        c[3] = (m11 * yp - m21 * xp) / det
        c[0] -= fx * k
        c[2] -= fy * k
        c[4] -= (c[1] * fx + c[3] * fy) * k * k
    else:
        raise ValueError(name)


class _Field:
    """The 2.5D space charge of one calculator."""

    def __init__(self, nx, ny, nz, keep_ratio=False):
        self.nx, self.ny, self.nz, self.keep, self.ratio = nx, ny, nz, keep_ratio, 1.0

    def _limits(self, c, pipe):
        lo = [float(c[k].min()) for k in (0, 2, 4)]
        hi = [float(c[k].max()) for k in (0, 2, 4)]
        if pipe is not None:
            lo[0], hi[0], lo[1], hi[1] = pipe
            return lo, hi
        r = (hi[0] - lo[0]) / (hi[1] - lo[1])
        if self.keep or abs(r - self.ratio) < 0.25 * self.ratio:
            i, f = (1, r / self.ratio) if r > self.ratio else (0, self.ratio / r)
            mid, half = 0.5 * (hi[i] + lo[i]), 0.5 * (hi[i] - lo[i]) * f
            lo[i], hi[i] = mid - half, mid + half
        if not self.keep:
            self.ratio = (hi[0] - lo[0]) / (hi[1] - lo[1])
        return lo, hi

    @staticmethod
    def _weights(t, n):
        i = (t + 0.5).to(torch.int64).clamp(1, n - 2)
        f = t - i
        return i, (0.5 * (0.5 - f) ** 2, 0.75 - f * f, 0.5 * (0.5 + f) ** 2), (f - 0.5, -2.0 * f, f + 0.5)

    def _line(self, z, zmin, dz):
        """Cells and weights of the periodic line density."""
        if self.nz == 1:
            i = torch.zeros_like(z, dtype=torch.int64)
            return (i, i), (torch.ones_like(z), torch.zeros_like(z))
        u = (z - zmin) / dz - 0.5
        i = torch.floor(u)
        w = u - i
        i = i.to(torch.int64)
        return (i % self.nz, (i + 1) % self.nz), (1.0 - w, w)

    def kick(self, c, length, macro, denoise=None, pipe=None, circle=None, pipe_radius=None):
        """macro: the macrosize or a tensor of them.  pipe: (limits, points,
        modes) of a circular boundary of radius `circle`."""
        nx, ny, nz = self.nx, self.ny, self.nz
        beta, gamma, _ = _kinematics()
        x, y, z = c[0], c[2], c[4]
        lo, hi = self._limits(c, pipe[0] if pipe else None)
        dx, dy, dz = (hi[0] - lo[0]) / (nx - 1), (hi[1] - lo[1]) / (ny - 1), (hi[2] - lo[2]) / nz
        ix, wx, gx = self._weights((x - lo[0]) / dx, nx)
        iy, wy, gy = self._weights((y - lo[1]) / dy, ny)
        inside = None
        if pipe:
            inside = (x >= lo[0]) & (x <= hi[0]) & (y >= lo[1]) & (y <= hi[1])
        each = macro if torch.is_tensor(macro) else torch.full_like(x, macro)
        rho = torch.zeros(nx * ny, dtype=torch.float64, device=x.device)
        for a in range(3):
            for b in range(3):
                v = wx[a] * wy[b] * each
                rho.index_add_(0, (ix + (a - 1)) * ny + (iy + (b - 1)), v if inside is None else v * inside)
        (z0, z1), (v0, v1) = self._line(z, lo[2], dz)
        lam = torch.zeros(nz, dtype=torch.float64, device=x.device)
        lam.index_add_(0, z0, v0 * each).index_add_(0, z1, v1 * each)
        rho = rho.view(nx, ny)
        if denoise is not None:
            total = float(rho.sum())
            out = denoise(rho * (nx * ny / total)).clamp(min=0.0)
            rho = out * (total / out.sum())
        i = torch.arange(2 * nx, device=x.device, dtype=torch.float64)
        j = torch.arange(2 * ny, device=x.device, dtype=torch.float64)
        r2 = ((torch.minimum(i, 2 * nx - i) * dx) ** 2)[:, None] + ((torch.minimum(j, 2 * ny - j) * dy) ** 2)[None]
        r2[0, 0] = 1.0
        spec = torch.fft.rfft2(rho, s=(2 * nx, 2 * ny)) * torch.fft.rfft2(-0.5 * torch.log(r2))
        phi = torch.fft.irfft2(spec, s=(2 * nx, 2 * ny))[:nx, :ny].contiguous()
        if pipe:
            phi = self._grounded(phi, lo, dx, dy, pipe)
        flat = phi.reshape(-1)
        ex, ey = torch.zeros_like(x), torch.zeros_like(x)
        for a in range(3):
            for b in range(3):
                p = flat[(ix + (a - 1)) * ny + (iy + (b - 1))]
                ex += gx[a] * wy[b] * p
                ey += wx[a] * gy[b] * p
        total = rho.sum() if pipe_radius is not None else lam.sum()
        f = -(v0 * lam[z0] + v1 * lam[z1]) * (2.0 * length * R_CLASSICAL / (beta ** 2 * gamma ** 3) / (dz * total))
        if circle is not None:
            f = f * (x * x + y * y < circle * circle)
        if pipe_radius is not None:
            self._longitudinal(c, rho, lam, lo, dx, dz, (z0, z1), (v0, v1), length, pipe_radius)
        c[1] += ex / dx * f
        c[3] += ey / dy * f

    def _grounded(self, phi, lo, dx, dy, pipe):
        """phi less the free-space harmonics fitted to it on the boundary."""
        _, (bx, by), modes = pipe
        bx, by = (torch.tensor(v, dtype=torch.float64, device=phi.device) for v in (bx, by))
        scale = float((bx * bx + by * by).sqrt().max())

        def harmonics(px, py):
            w = torch.complex(px, py) / scale
            rows = [torch.ones_like(px)]
            for m in range(1, modes + 1):
                rows += [(w ** m).real, (w ** m).imag]
            return torch.stack(rows, -1)

        i, wx, _ = self._weights((bx - lo[0]) / dx, self.nx)
        j, wy, _ = self._weights((by - lo[1]) / dy, self.ny)
        on = sum(wx[a] * wy[b] * phi[i + (a - 1), j + (b - 1)] for a in range(3) for b in range(3))
        coef = torch.linalg.lstsq(harmonics(bx, by), on[:, None]).solution[:, 0]
        gx = lo[0] + dx * torch.arange(self.nx, device=phi.device, dtype=torch.float64)
        gy = lo[1] + dy * torch.arange(self.ny, device=phi.device, dtype=torch.float64)
        return phi - harmonics(*torch.meshgrid(gx, gy, indexing="ij")) @ coef

    def _longitudinal(self, c, rho, lam, lo, dx, dz, zi, zw, length, pipe_radius):
        """dE from the slope of the line density (a parabola through three
        cells) and the radius of the beam on the grid."""
        beta, gamma, _ = _kinematics()
        nx, ny, nz = self.nx, self.ny, self.nz
        gx = lo[0] + dx * torch.arange(max(nx, ny), device=rho.device, dtype=torch.float64)
        wx, wy = rho.sum(1), rho.sum(0)
        total = rho.sum()
        xc, yc = (wx * gx[:nx]).sum() / total, (wy * gx[:ny]).sum() / total
        x2, y2 = (wx * gx[:nx] ** 2).sum() / total, (wy * gx[:ny] ** 2).sum() / total
        a2 = 2.0 * ((x2 - xc * xc).abs() + (y2 - yc * yc).abs())
        k = torch.arange(nz, device=rho.device)
        i0 = (k - 1).clamp(0, nz - 3)
        p, q, r = lam[i0], lam[i0 + 1], lam[i0 + 2]
        t = (k - i0).to(torch.float64)  # 0, 1 or 2
        slope = (-1.5 * p + 2.0 * q - 0.5 * r + t * (p - 2.0 * q + r)) / (dz * dz)
        ez = zw[0] * slope[zi[0]] + zw[1] * slope[zi[1]]
        d2 = (c[0] - xc) ** 2 + (c[2] - yc) ** 2
        inner = 1.0 + 2.0 * torch.log(pipe_radius / a2.sqrt()) - d2 / a2
        outer = 2.0 * math.log(pipe_radius) - torch.log(d2)
        c[5] += ez * torch.where(d2 <= a2, inner, outer) * (-length * R_CLASSICAL * MASS / gamma ** 2)


_CHANNELS = ((1, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 64), (64, 64), (128, 64), (64, 64),
             (96, 32), (32, 32), (48, 16), (16, 16))


def _parameters(requires_grad=False):
    """The network's layers from its parameter file, 3x3 weights rounded to
    BF16: [(weight, bias)] and the output layer."""
    p = np.load(os.path.join(_PKG, "orbit_gb300", "data", "denoiser_128x128.npy"))
    p = torch.from_numpy(p).to(_device())
    layers, at = [], 0
    for cin, cout in _CHANNELS:
        w = p[at:at + cin * cout * 9].bfloat16().double().view(cout, cin, 3, 3)
        at += cin * cout * 9
        layers.append((w, p[at:at + cout].double()))
        at += cout
    layers.append((p[at:at + 16].double().view(1, 16, 1, 1), p[at + 16:at + 17].double()))
    if requires_grad:
        layers = [(w.clone().requires_grad_(), b.clone().requires_grad_()) for w, b in layers]
    return layers


def _network(x, layers):
    F = torch.nn.functional

    def conv(h, k):
        return torch.relu(F.conv2d(h, layers[k][0], layers[k][1], padding=1))

    def up(h, skip):
        return torch.cat([F.interpolate(h, scale_factor=2, mode="nearest"), skip], 1)

    s1 = conv(conv(x, 0), 1)
    s2 = conv(conv(F.avg_pool2d(s1, 2), 2), 3)
    s3 = conv(conv(F.avg_pool2d(s2, 2), 4), 5)
    h = conv(conv(F.avg_pool2d(s3, 2), 6), 7)
    h = conv(conv(up(h, s3), 8), 9)
    h = conv(conv(up(h, s2), 10), 11)
    h = conv(conv(up(h, s1), 12), 13)
    return x + F.conv2d(h, layers[14][0], layers[14][1])


def _exact_line(c, ops, field, macro, denoise=None):
    for op in ops:
        if op[0] == "sc":
            field.kick(c, op[1], macro, denoise)
        else:
            _map(op, c)
    return c


def _exact_diag(case, seed):
    c, _, _ = _beam(case, seed)
    n, order = case["n"], case["order"]
    avg = c.mean(1)
    e = c - avg[:, None]
    corr = e @ e.T / n

    def emittance(i):
        xx, pp, xp = corr[i, i], corr[i + 1, i + 1], corr[i, i + 1]
        xd, pd, dd = corr[i, 5], corr[i + 1, 5], corr[5, 5]
        a, b, m = xx - xd * xd / dd, pp - pd * pd / dd, xp - xd * pd / dd
        return a, (a * b - m * m).abs().sqrt()

    (ax, exx), (ay, eyy) = emittance(0), emittance(2)
    bx, by = (ax / exx).sqrt(), (ay / eyy).sqrt()
    mom = torch.zeros(order + 1, order + 1, dtype=torch.float64, device=c.device)
    for j in range(order):
        for i in range(order + 1 - j):
            mom[i, j] = (e[0] ** i * e[2] ** j).sum() / (bx ** i * by ** j) / n
    mom[2, order] += (e[0] ** 2 * e[2] ** order).sum()  # added once per particle, not normalised
    mom[0, 0], mom[1, 0], mom[0, 1] = 1.0, avg[0], avg[2]
    return {"avg": avg.cpu().numpy(), "corr": corr.cpu().numpy(), "emit": torch.stack([exx, eyy]).cpu().numpy(),
            "moments": mom.cpu().numpy()}


def _exact_train(case, seed):
    x, t = _images(case, seed)
    layers = _parameters(requires_grad=True)
    y = _network(x.double(), layers)
    loss = ((y - t.double()) ** 2).mean()
    grads = torch.autograd.grad(loss, [p for wb in layers for p in wb])
    return {"loss": float(loss.detach()), "grads": torch.cat([g.reshape(-1) for g in grads]).cpu().numpy(), "y": y.detach()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "diag":
        return _exact_diag(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "batch":
        out = []
        for k, (n, grid, k1, protons) in enumerate(_scan(case, seed)):
            c = _exact_line(_gauss(n, _gen(seed, 1 + k)), _fodo_ops(case["cells"], k1), _Field(*grid), protons / n)
            out += [c[0], c[1], c[3], c[4]]
        return out
    c, macro, msize = _beam(case, seed)
    field = _Field(case["nx"], case["ny"], case["nz"], keep_ratio=kind == "rb")
    if kind == "kick":
        field.kick(c, KICK_LENGTH, macro if msize is None else msize)
    elif kind == "rb":
        field.kick(c, KICK_LENGTH, macro, pipe_radius=PIPE_RADIUS)
    elif kind == "boundary":
        np_, r = case["points"], PIPE / 2.0
        angle = [2.0 * math.pi * i / np_ for i in range(np_)]
        pts = [r * math.sin(a) for a in angle], [r * math.cos(a) for a in angle]
        limits = (min(pts[0]), max(pts[0]), min(pts[1]), max(pts[1]))
        field.kick(c, KICK_LENGTH, macro, pipe=(limits, pts, case["modes"]), circle=r)
    else:
        denoise = None
        if kind == "fodo" and case["form"] == "learned":
            layers = _parameters()
            denoise = lambda rho: _network(rho[None, None], layers)[0, 0]  # noqa: E731
        ops = _ring_ops(case["cells"]) if kind == "ring" else _fodo_ops(case["cells"], case["kq"])
        _exact_line(c, ops, field, macro, denoise)
    return [c[k] for k in range(6)]
