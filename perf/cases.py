"""What a program does with this library, as cases that can be timed and compared.

A simulation program keeps a solver per scene and advances it frame by frame through
``step_state_range_ptr`` / ``step_state_ranges_ptr``: the fluid state it holds in pinned host
memory goes in, a few substeps run, the new state comes back.  A learning program records a
rollout and asks for its gradients (``diff_forward`` / ``diff_backward``).  A program with its
own solver takes only the neighbour lists, from device memory to device memory
(``vtp_ugns_neighbors_noalloc``).  Configurations are the defaults; scenes are the dam breaks,
mixtures and blocks of ``vtp.scenes`` over the sizes their users run.

``exact`` restates PBF, DFSPH and the neighbour search in plain torch, in 64 bits; the gradients
are torch.autograd's through that restatement.
"""
from __future__ import annotations

import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "vt-physics_b200"))
from vtp import diff, scenes, solver  # noqa: E402
from vtp._lib import check, lib  # noqa: E402

# ------------------------------------------------------------------ the cases


def listed() -> list:
    return [
        # An interactive toy scene: every launch counts.  Odd particle count.
        {"name": "pbf_2k", "kind": "pbf", "n": 2000, "drop": 37, "jitter": 0.1, "form": "reference", "steps": 4},
        # The benchmark's dam break (20 x 40 x 20 lattice) at mass-1 particles, one 60 Hz frame.
        {"name": "pbf_16k", "kind": "pbf", "n": 16000, "drop": 0, "jitter": 0.1, "form": "reference", "steps": 4},
        # A film-size PBF scene with the standard (poly6 / spiky) constraint.
        {"name": "pbf_250k", "kind": "pbf", "n": 250000, "drop": 101, "jitter": 0.1, "form": "standard", "steps": 4},
        # A small DFSPH dam break, four fixed steps of 1 ms.
        {"name": "dfsph_8k", "kind": "dfsph", "n": 8000, "drop": 37, "jitter": 0.05, "cfl": 0.0, "steps": 4},
        # Two fluid objects thrown at each other, surface tension on, per-object residuals.
        {"name": "dfsph_blocks", "kind": "blocks", "side": 25, "jitter": 0.05, "tension": 0.001, "steps": 2},
        # The headline scene: 1M fluid particles, the benchmark's adaptive step, one substep a frame.
        {"name": "dfsph_1m", "kind": "dfsph_1m", "jitter": 0.05, "cfl": 0.4, "steps": 1},
        # A three-phase mixture whose fractions are read back for display.
        {"name": "imm_55k", "kind": "mixture", "solver": "IMM", "side": 48, "jitter": 0.05, "steps": 4},
        # The conformation-tensor mixture at the benchmark's size, fractions read back.
        {"name": "immct_500k", "kind": "mixture", "solver": "IMMCT", "side": 100, "jitter": 0.05, "steps": 2},
        # Many independent scenes in one solver (parameter sweeps, training data).
        {"name": "batch_dfsph", "kind": "batch", "solver": "DFSPH", "scenes": 16, "n_min": 4000, "n_max": 32000,
         "jitter": 0.05, "steps": 2},
        # Neighbour lists alone, device to device, for a host with its own solver.
        {"name": "lists_400k", "kind": "lists", "n": 400000, "drop": 333, "jitter": 0.2, "max_nbr": 60},
        # A gradient of a PBF rollout (the differentiable benchmark scene, checkpoints kept).
        {"name": "grad_pbf_64k", "kind": "grad", "solver": "PBF", "side": 40, "steps": 10, "every": 5},
        # A gradient of a DFSPH rollout.
        {"name": "grad_dfsph_27k", "kind": "grad", "solver": "DFSPH", "side": 30, "steps": 4, "every": 2},
    ]


def draw(rng) -> dict:
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["pbf", "pbf", "dfsph", "dfsph", "blocks", "mixture", "batch", "lists", "grad"])
    if kind == "pbf":
        return {"kind": kind, "n": size(1000, 250000), "drop": rng.randrange(400), "jitter": rng.uniform(0.02, 0.12),
                "form": rng.choice(["reference", "standard"]), "steps": rng.choice([1, 2, 4])}
    if kind == "dfsph":
        return {"kind": kind, "n": size(1000, 300000), "drop": rng.randrange(400), "jitter": rng.uniform(0.03, 0.06),
                "cfl": rng.choice([0.0, 0.4]), "steps": rng.choice([1, 2])}
    if kind == "blocks":
        return {"kind": kind, "side": rng.randrange(8, 45), "jitter": rng.uniform(0.03, 0.06),
                "tension": rng.choice([0.0, 0.001]), "steps": rng.choice([1, 2])}
    if kind == "mixture":
        return {"kind": kind, "solver": rng.choice(["IMM", "IMMCT"]), "side": rng.randrange(16, 81),
                "jitter": rng.uniform(0.03, 0.06), "steps": rng.choice([1, 2, 4])}
    if kind == "batch":
        lo = size(1000, 8000)
        return {"kind": kind, "solver": rng.choice(["PBF", "DFSPH"]), "scenes": rng.randrange(2, 25), "n_min": lo,
                "n_max": lo * rng.choice([1, 2, 4, 8]), "jitter": rng.uniform(0.03, 0.06), "steps": rng.choice([1, 2])}
    if kind == "lists":
        return {"kind": kind, "n": size(1000, 800000), "drop": rng.randrange(400), "jitter": rng.uniform(0.02, 0.4),
                "max_nbr": rng.choice([48, 60, 64, 96])}
    return {"kind": kind, "solver": rng.choice(["PBF", "DFSPH"]), "side": rng.randrange(8, 37),
            "steps": rng.randrange(3, 9), "every": rng.randrange(2, 6)}


# ------------------------------------------------------------------ inputs


def _fluid(sc):
    return [o for o in sc.objects if o.material == scenes.EPM_FLUID]


def _noise(sc, seed, speed):
    """Per-particle velocity noise of `speed` m/s on top of the objects' start velocities."""
    rng = np.random.default_rng(seed)
    for o in _fluid(sc):
        o.velocity = (np.asarray(o.velocity_start, np.float32) +
                      speed * rng.standard_normal(o.pos.shape, np.float32)).astype(np.float32)
    return sc


def _scene(case, seed):
    kind = case["kind"]
    if kind in ("pbf", "dfsph"):
        sc = scenes.dam_break(kind.upper(), case["n"], seed, jitter_amp=case["jitter"],
                              spacing=0.1 if kind == "pbf" else None)
        o = sc.objects[0]
        o.pos = o.pos[: max(64, o.n - case["drop"])]
        o.velocity_start = (2.0 if kind == "pbf" else 1.0, 0.0, 0.0)   # the fluid is on its way
        return _noise(sc, seed, 0.1 if kind == "pbf" else 0.02)
    if kind == "dfsph_1m":
        return _noise(scenes.dfsph_1m(seed, case["jitter"]), seed, 0.02)
    if kind == "blocks":
        return _noise(scenes.colliding_blocks(seed, case["tension"], n_side=case["side"], jitter_amp=case["jitter"]),
                      seed, 0.02)
    if kind == "mixture":
        sc = scenes.layered_mixture(case["solver"], case["side"], seed, case["jitter"])
        req = sc.config[case["solver"]]["Required"]
        req["divFreeThreshold"] = req["incompThreshold"] = 1e-3   # as the benchmark's mixture
        if case["solver"] == "IMMCT":
            # A frame starts from the caller's positions while the phase velocities and the
            # conformation tensor stay in the solver: a thin polymer solution with the template's
            # relaxation time keeps that bounded however many frames are asked for.
            req.update(solventViscosity=0.02, relaxationTime=0.001, solutionBasicViscosity=8e-6,
                       solutionMaxViscosity=1.2e-5)
        return _noise(sc, seed, 0.005)
    if kind == "grad":   # the differentiable benchmark scenes with another side length
        side, pbf = case["side"], case["solver"] == "PBF"
        sp, layers = (0.02, 2) if pbf else (0.01, 3)
        off, w = 10 * sp, side * sp
        pos = scenes.cube(sp / 2, (off,) * 3, (w,) * 3)
        wall = scenes.box(sp / 2, (0.0,) * 3, (w + 2 * off,) * 3, layers)
        make = scenes.pbf_config if pbf else scenes.dfsph_config
        cfg = make(dt=1.0 / 240.0 if pbf else 1e-3, r=sp / 2, lb=(-5 * sp,) * 3, size=(w + 2 * off + 10 * sp,) * 3)
        sc = scenes.Scene(case["solver"], cfg, [scenes.SceneObject("fluid", pos, scenes.EPM_FLUID),
                                                scenes.SceneObject("box", wall, scenes.EPM_BOUNDARY)])
        return _noise(sc, seed, 0.1)
    raise ValueError(kind)


def _batch(case, seed):
    rng = np.random.default_rng(seed)
    # the sizes are the case's and only their order the seed's: every seed is the same amount of work
    ns = rng.permutation(np.exp(np.linspace(math.log(case["n_min"]), math.log(case["n_max"]), case["scenes"])))
    return [_noise(scenes.dam_break(case["solver"], int(n), seed + k, gravity_y=float(rng.uniform(-12, -8)),
                                    jitter_amp=case["jitter"], spacing=0.1 if case["solver"] == "PBF" else None),
                   seed + k, 0.02) for k, n in enumerate(ns)]


def _extra(case):
    extra = {}
    if case.get("cfl"):
        extra["cfl"] = case["cfl"]
    if case.get("form") == "standard":
        extra["pbfFormulation"] = "standard"
    return extra or None


def _cloud(case, seed):
    """Positions of a jittered block, h, and the box the lists are searched in."""
    k = max(2, round(case["n"] ** (1 / 3)))
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(k, dtype=np.float32)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (0.01 * (g + case["jitter"] * rng.uniform(-1, 1, g.shape))).astype(np.float32)
    return pos[: max(64, len(pos) - case["drop"])], 0.02, -0.05, 0.01 * k + 0.1


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def prepare(case, seed) -> dict:
    kind = case["kind"]
    if kind == "lists":
        pos, h, lb, size = _cloud(case, seed)
        n = len(pos)
        dev = torch.device("cuda")
        return {"kind": kind, "pos": torch.from_numpy(pos).to(dev), "h": h, "lb": (C.c_float * 3)(lb, lb, lb),
                "size": (C.c_float * 3)(size, size, size), "max_nbr": case["max_nbr"],
                "count": torch.empty(n, dtype=torch.int32, device=dev),
                "nbr": torch.empty((n, case["max_nbr"]), dtype=torch.int32, device=dev)}
    if kind == "batch":
        group = _batch(case, seed)
        s, ranges = solver.solver_from_scenes(group)
        spans = [(a, sc.n_fluid) for (a, _), sc in zip(ranges, group)]
    else:
        group = [_scene(case, seed)]
        s = solver.solver_from_scene(group[0], extra=_extra(case))
        spans = [(0, group[0].n_fluid)]
    s.initialize()
    objs = [o for sc in group for o in _fluid(sc)]
    state = {"kind": kind, "solver": s, "spans": spans, "steps": case["steps"],
             "pos": _pinned(np.concatenate([o.pos for o in objs])),
             "vel": _pinned(np.concatenate([o.velocity for o in objs]))}
    if kind == "grad":
        n, nf = group[0].n_total, group[0].n_fluid
        for name, seed_of in (("gpos", 1), ("gvel", 2)):
            state[name] = np.zeros((n, 3), np.float32)
            state[name][:nf] = np.random.default_rng([seed, seed_of]).standard_normal((nf, 3), np.float32)
        state["every"] = case["every"]
    else:
        state["pos_out"], state["vel_out"] = (torch.empty(state["pos"].shape, pin_memory=True) for _ in range(2))
        state["fractions"] = kind == "mixture"
    return state


def run(state):
    kind = state["kind"]
    if kind == "lists":
        pos = state["pos"]
        check(lib().vtp_ugns_neighbors_noalloc(pos.data_ptr(), pos.shape[0], state["lb"], state["size"], state["h"],
                                               state["max_nbr"], state["count"].data_ptr(), state["nbr"].data_ptr(),
                                               torch.cuda.current_stream().cuda_stream), "neighbours")
        return {"count": state["count"], "nbr": state["nbr"]}
    s, p, v = state["solver"], state["pos"], state["vel"]
    if kind == "grad":
        nf = state["spans"][0][1]
        s.set_state_range_ptr(0, nf, p.data_ptr(), v.data_ptr())
        diff.diff_forward(s, state["steps"], state["every"])
        pos = s.get_field("pos")
        dpos, dvel, dparam = diff.diff_backward(s, state["gpos"], state["gvel"])
        return {"pos": pos, "dpos": dpos, "dvel": dvel, "dparam": dparam}
    po, vo = state["pos_out"], state["vel_out"]
    if len(state["spans"]) > 1:
        s.step_state_ranges_ptr(state["spans"], p.data_ptr(), v.data_ptr(), state["steps"], po.data_ptr(), vo.data_ptr())
    else:
        first, count = state["spans"][0]
        s.step_state_range_ptr(first, count, p.data_ptr(), v.data_ptr(), state["steps"], po.data_ptr(), vo.data_ptr())
    out = {"pos": po, "vel": vo}
    if state["fractions"]:
        out["fractions"] = s.get_field("vol_frac")
    return out


def _counts(case):
    """(fluid, boundary) particles of a case, as its scene has them."""
    if case["kind"] == "batch":
        group = _batch(case, 0)
        return sum(sc.n_fluid for sc in group), sum(sc.n_boundary for sc in group)
    sc = _scene(case, 0)
    return sc.n_fluid, sc.n_boundary


def work(case) -> dict:
    """Inputs read once and outputs written once; about 30 neighbours a particle, 30 operations a
    neighbour and pass, and the passes a substep has when its solves take one iteration each."""
    kind = case["kind"]
    if kind == "lists":
        n = len(_cloud(case, 0)[0])
        return {"bytes": n * (12 + 4 + 4 * case["max_nbr"]), "flops": n * 27 * 8 * 9}
    nf, nb = _counts(case)
    state = 48 * nf + 12 * nb   # position and velocity in and out, boundary positions in
    passes = {"PBF": 9, "DFSPH": 6, "IMM": 9, "IMMCT": 11}[
        case.get("solver") or ("PBF" if kind == "pbf" else "DFSPH")]
    flops = nf * 30 * 30 * passes * case["steps"]
    if kind == "grad":
        return {"bytes": 2 * state, "flops": 3 * flops}
    if kind == "mixture":
        state += 4 * (2 if case["solver"] == "IMMCT" else 3) * (nf + nb)
    return {"bytes": state, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits

F32 = np.float32


def _pairs(x, rows, h, lb):
    """(i, j), i < rows, of the pairs with 0 < |x_i - x_j| <= h."""
    c = torch.floor((x.detach() - lb) / h).long() + 1
    dims = c.max(0).values + 2
    key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    order = torch.argsort(key)
    skey = key[order]
    ii, jj = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = key[:rows] + (dz * dims[1] + dy) * dims[0] + dx
                lo, hi = torch.searchsorted(skey, k), torch.searchsorted(skey, k, right=True)
                cnt = hi - lo
                i = torch.repeat_interleave(torch.arange(rows, device=x.device), cnt)
                at = torch.arange(i.numel(), device=x.device) - (torch.cumsum(cnt, 0) - cnt)[i] + lo[i]
                j = order[at]
                d2 = (x.detach()[i] - x.detach()[j]).square().sum(1)
                m = (d2 > 0) & (d2 <= h * h)
                ii.append(i[m])
                jj.append(j[m])
    return torch.cat(ii), torch.cat(jj)


def _w(r, h):
    q = r / h
    s = 8 / math.pi / h ** 3
    return torch.where(q > 1, 0 * q, s * torch.where(q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, 2 * (1 - q) ** 3))


def _g(r, h):
    """gradW = _g * (x_i - x_j)."""
    q = r / h
    s = 8 / math.pi / h ** 3
    return torch.where(q > 1, 0 * q, s * torch.where(q <= 0.5, 6 * q * (3 * q - 2), -6 * (1 - q) ** 2)) / (r * h)


def _sum(v, i, n):
    return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add(0, i, v)


class _Exact:
    """One scene in 64 bits: `x`, `v` of the fluid rows, the boundary behind them."""

    def __init__(self, sc, extra):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        req, opt = sc.config[sc.solver]["Required"], sc.config[sc.solver]["Optional"]
        f = lambda v: float(F32(v))  # noqa: E731  (the library reads its parameters as floats)
        self.extra = extra or {}
        self.solver, self.r, self.dt = sc.solver, f(req["particleRadius"]), f(req["timeStep"])
        self.h, self.vol = 4 * self.r, float(F32(2 * self.r) ** F32(3))
        self.rho, self.rho_b = f(req["fPartRestDensity"]), f(req["bPartRestDensity"])
        self.m = float(F32(self.rho) * F32(self.vol))
        self.lb = f(req["simSpaceLB"][0])
        self.grav = torch.tensor([f(g) for g in opt["gravity"]], dtype=torch.float64, device=dev)
        self.req = req
        fl = _fluid(sc)
        self.sizes = [o.n for o in fl]
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev, torch.float64)  # noqa: E731
        self.x, self.v = t(np.concatenate([o.pos for o in fl])), t(np.concatenate([o.velocity for o in fl]))
        self.xb = t(np.concatenate([o.pos for o in sc.objects if o.material == scenes.EPM_BOUNDARY]))
        self.nf, self.nb = len(self.x), len(self.xb)
        self.standard = self.extra.get("pbfFormulation") == "standard"
        i, j = _pairs(self.xb, self.nb, self.h, self.lb)
        r = (self.xb[i] - self.xb[j]).norm(dim=1)
        zero = torch.zeros(1, dtype=torch.float64, device=dev)
        self.vb = 1 / (self._pbf_w(zero) + _sum(self._pbf_w(r), i, self.nb))

    def _pbf_w(self, r):
        if not self.standard:
            return _w(r, self.h)
        return 315 / (64 * math.pi * self.h ** 9) * (self.h ** 2 - r ** 2).clamp(min=0) ** 3

    def _pbf_g(self, r):
        if not self.standard:
            return _g(r, self.h)
        return -45 / (math.pi * self.h ** 6) * (self.h - r).clamp(min=0) ** 2 / r

    def pbf(self, x, v, xsph):
        n, h, rho = self.nf, self.h, self.rho
        v = v + self.grav * self.dt
        x = x + v * self.dt
        i, j = _pairs(torch.cat([x, self.xb]), n, h, self.lb)
        mass = torch.cat([torch.full((n,), self.m, dtype=x.dtype, device=x.device), self.rho_b * self.vb])
        vol = torch.cat([torch.full((n,), self.vol, dtype=x.dtype, device=x.device), self.vb])
        eps = 100.0 if self.standard else float(F32(1e-6))
        for _ in range(self.req["iterationNum"]):
            full = torch.cat([x, self.xb])
            d = full[i] - full[j]
            r = d.norm(dim=1)
            g = self._pbf_g(r)
            grad = (g * mass[j] if self.standard else g)[:, None] * d / rho
            dens = self.m * self._pbf_w(torch.zeros(1, dtype=x.dtype, device=x.device)) + \
                _sum(mass[j] * self._pbf_w(r), i, n)
            err = dens.clamp(min=rho) / rho - 1
            lam = -err / (_sum(grad.square().sum(1), i, n) + _sum(grad, i, n).square().sum(1) + eps)
            both = torch.cat([lam, torch.zeros_like(self.vb)])
            c = both[i] * mass[j] + both[j] * mass[i] if self.standard else both[i] + both[j]
            dx = _sum((c * g)[:, None] * d, i, n) / rho
            x, v = x + dx, v + dx / self.dt
        full, vel = torch.cat([x, self.xb]), torch.cat([v, torch.zeros_like(self.xb)])
        w = self._pbf_w((full[i] - full[j]).norm(dim=1))
        a = _sum((xsph * vol[j] * w)[:, None] * (vel[j] - vel[i]), i, n)
        return x + a * self.dt, v + a

    def _solve(self, v, i, j, d, g, ratio, alpha, dt, threshold):
        n, zero = self.nf, torch.zeros_like(self.xb)
        vol = torch.cat([torch.full((n,), self.vol, dtype=v.dtype, device=v.device), self.vb])
        for _ in range(101):
            full = torch.cat([v, zero])
            delta = (ratio - 1 + dt * _sum(vol[j] * g * (d * (full[i] - full[j])).sum(1), i, n)).clamp(min=0)
            kap = torch.cat([delta / alpha / dt ** 2 / self.vol, torch.zeros_like(self.vb)])
            c = dt * self.vol / self.m * vol[j] * (kap[i] + kap[j]) * g
            v = v - _sum(c[:, None] * d, i, n)
            if float(torch.stack([o.mean() for o in delta.detach().split(self.sizes)]).mean()) < threshold:
                break
        return v

    def dfsph(self, x, v, nu):
        n, h, dt = self.nf, self.h, self.dt
        if self.extra.get("cfl"):
            fast = float(v.detach().norm(dim=1).max())
            dt = min(dt, self.extra["cfl"] * 2 * self.r / fast) if fast > 0 else dt
        full = torch.cat([x, self.xb])
        i, j = _pairs(full, n, h, self.lb)
        d = full[i] - full[j]
        r = d.norm(dim=1)
        g = _g(r, h)
        vol = torch.cat([torch.full((n,), self.vol, dtype=x.dtype, device=x.device), self.vb])
        ratio = self.vol * 8 / math.pi / h ** 3 + _sum(vol[j] * _w(r, h), i, n)
        gd = g[:, None] * d
        fluid = (j < n).to(x.dtype)
        alpha = _sum(vol[j][:, None] * gd, i, n).square().sum(1) / self.m + float(F32(1e-6)) + \
            _sum(fluid * gd.square().sum(1) * vol[j] ** 2 / self.m, i, n)
        alpha = alpha.clamp(min=float(F32(1e-6)))
        v = self._solve(v, i, j, d, g, ratio, alpha, dt, float(F32(self.req["divFreeThreshold"])))
        k = j < n
        a, b, e, q = i[k], j[k], d[k], g[k]
        pi = nu * self.m / self.rho * ((v[a] - v[b]) * e).sum(1) / (e.square().sum(1) + 0.001 * h * h)
        acc = self.grav + _sum((10 * pi * q)[:, None] * e, a, n)
        gamma = float(F32(self.req["surfaceTensionCoefficient"]))
        if gamma:
            nrm = _sum((h * self.m / self.rho * q)[:, None] * e, a, n)
            l = e.norm(dim=1)
            cub = (h - l) ** 3 * l ** 3
            coh = 32 / math.pi / h ** 9 * torch.where(2 * l > h, cub, 2 * cub - h ** 6 / 64)
            acc = acc - gamma * self.m * _sum((self.m * coh / l)[:, None] * e + nrm[a] - nrm[b], a, n)
        v = v + acc * dt
        v = self._solve(v, i, j, d, g, ratio, alpha, dt, float(F32(self.req["incompThreshold"])))
        return x + v * dt, v

    def param(self):
        return float(F32(self.req["XSPH_k" if self.solver == "PBF" else "fPartRestViscosity"]))

    def step(self, x, v, p):
        return self.pbf(x, v, p) if self.solver == "PBF" else self.dfsph(x, v, p)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mixture", "lists"):
        return None   # the mixtures' substep is not restated here; lists are whole numbers
    if kind == "batch":
        got = []
        for sc in _batch(case, seed):
            e = _Exact(sc, None)
            x, v = e.x, e.v
            for _ in range(case["steps"]):
                x, v = e.step(x, v, e.param())
            got.append((x, v))
        return {"pos": torch.cat([x for x, _ in got]), "vel": torch.cat([v for _, v in got])}
    e = _Exact(_scene(case, seed), _extra(case))
    x, v = e.x, e.v
    if kind != "grad":
        for _ in range(case["steps"]):
            x, v = e.step(x, v, e.param())
        return {"pos": x, "vel": v}
    x0, v0 = x.clone().requires_grad_(), v.clone().requires_grad_()
    p = torch.tensor(e.param(), dtype=x.dtype, device=x.device, requires_grad=True)
    x, v = x0, v0
    for _ in range(case["steps"]):
        x, v = checkpoint(e.step, x, v, p, use_reentrant=False)
    loss = 0
    for name, seed_of in ((x, 1), (v, 2)):
        gr = np.random.default_rng([seed, seed_of]).standard_normal((e.nf, 3), np.float32)
        loss = loss + (name * torch.from_numpy(gr).to(x)).sum()
    loss.backward()
    pad = torch.zeros_like(e.xb)
    return {"pos": torch.cat([x.detach(), e.xb]), "dpos": torch.cat([x0.grad, pad]),
            "dvel": torch.cat([v0.grad, pad]), "dparam": float(p.grad)}
