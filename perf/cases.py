"""The work that programs built on this framework have it do, as measurable cases.

A pass is one rendered or recorded frame of a simulation: a few substeps
(``MpmPipeline.step``) and then what a program takes out of the state, either
the render data written into its own GPU buffers (``MpmState.prep_render``:
positions, deformations and velocity colors of every particle) or the
positions and velocities read back to the host.  The state goes on from pass
to pass, as a running simulation does.

``exact`` is the same frame in 64-bit torch: an MLS-MPM step over a dense grid,
written from the equations (quadratic B-splines, APIC transfers, the six
constitutive models, slip / stick / separate walls).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from nexus_b200 import scenes
from nexus_b200.models import BoundaryCondition, ParticleModel
from nexus_b200.mpm import (RENDER_VELOCITY, MpmPipeline, batched_collider_offsets, batched_state_from_scenes,
                            drive_kinematics, state_from_scene)
from nexus_b200.particles import ParticleBatch, box_walls, collider_array

def listed():
    return [
        # The smallest scene of the serving workload at the finest cell: 2k particles over a box of at
        # least 0.1 a side, so a particle in several cells; the result is read by the host.  Latency.
        {"name": "sparse_water_2k", "kind": "box", "material": "water", "n": 2048, "cells": 256, "steps": 4,
         "out": "read"},
        # A small interactive body: 16^3 particles, one substep a frame, rendered from the GPU.
        {"name": "cube_4k", "kind": "cube", "side": 16, "steps": 1, "out": "render"},
        # The benchmark's elastic cube (32,768 particles, dx = 1/64).
        {"name": "cube_32k", "kind": "cube", "side": 32, "steps": 10, "out": "render"},
        # Every constitutive model side by side, ragged block sizes, sticky floor and frictional walls.
        {"name": "materials_20k", "kind": "mixed", "side": 15, "steps": 8, "out": "read"},
        # A middle-sized serving request: sand in random positions.
        {"name": "sand_box_150k", "kind": "box", "material": "sand", "n": 150001, "cells": 128, "steps": 8,
         "out": "render"},
        # A large serving request: snow at the fine cell, random positions.
        {"name": "snow_box_500k", "kind": "box", "material": "snow", "n": 500000, "cells": 256, "steps": 8,
         "out": "render"},
        # The flagship scene of the benchmark: 1.5 M sand and 0.5 M water particles at dx = 1/256.
        {"name": "sand_water_2m", "kind": "column", "scale": 1.0, "steps": 8, "out": "render"},
        # The same scene at a quarter more per axis: 3.9 M particles.
        {"name": "sand_water_4m", "kind": "column", "scale": 1.25, "steps": 8, "out": "render"},
        # Batched scenes, half elastic, half sand, 4k-128k particles each, as the batched workload.
        {"name": "batch_48", "kind": "batch", "count": 48, "sizes": 7, "steps": 8, "out": "render"},
        # Bit-reproducible runs: the gather-form transfers in the reference's order of operations.
        {"name": "deterministic_100k", "kind": "box", "material": "sand", "n": 100003, "cells": 128, "steps": 4,
         "out": "render", "deterministic": True},
        # Scenes with driven bodies and a 20k-triangle floor, the velocities written every step.
        {"name": "coupled_6", "kind": "coupled", "count": 6, "steps": 6, "out": "render", "cpic": False},
        # The same with compatible-particle coupling (what a program with colliders runs by default).
        {"name": "coupled_cpic_4", "kind": "coupled", "count": 4, "steps": 6, "out": "render", "cpic": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["box", "box", "box", "cube", "mixed", "column", "batch", "deterministic", "coupled"])
    out = rng.choice(["render", "render", "read"])
    steps = rng.randint(1, 12)
    if kind == "box":
        return {"kind": "box", "material": rng.choice(["elastic", "neo_hookean", "sand", "sand_neo_hookean", "water", "snow"]),
                "n": _log_int(rng, 2048, 1000000), "cells": rng.choice([128, 256]), "steps": steps, "out": out}
    if kind == "cube":
        return {"kind": "cube", "side": rng.randint(9, 48), "steps": steps, "out": out}
    if kind == "mixed":
        return {"kind": "mixed", "side": rng.randint(6, 20), "steps": steps, "out": out}
    if kind == "column":
        return {"kind": "column", "scale": rng.randint(20, 115) / 100.0, "steps": rng.randint(1, 8), "out": "render"}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(2, 40), "sizes": rng.randint(100, 100000), "steps": rng.randint(1, 8),
                "out": "render"}
    if kind == "deterministic":
        return {"kind": "box", "material": rng.choice(["neo_hookean", "sand", "water"]), "n": _log_int(rng, 2048, 200000),
                "cells": 128, "steps": rng.randint(1, 6), "out": "render", "deterministic": True}
    return {"kind": "coupled", "count": rng.randint(1, 5), "steps": rng.randint(1, 6), "out": "render",
            "cpic": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _model(material):
    return {"elastic": (1000.0, ParticleModel.elastic(2.0e5, 0.25)),
            "neo_hookean": (1000.0, ParticleModel.elastic_neo_hookean(1.0e5, 0.3)),
            "sand": (2700.0, ParticleModel.sand_with_friction_angle(3.5e5, 0.3, 30.0)),
            "sand_neo_hookean": (2700.0, ParticleModel.sand_neo_hookean(3.5e5, 0.3)),
            "water": (1000.0, ParticleModel.water(1.0e5)),
            "snow": (400.0, ParticleModel.snow(1.4e5, 0.2))}[material]


def _in_motion(batch: ParticleBatch, rng: np.random.Generator) -> ParticleBatch:
    """The particles as a running simulation has them: falling and swirling,
    slightly and unevenly strained."""
    n = batch.n
    c = batch.pos.mean(axis=0, dtype=np.float64)
    r = batch.pos - c.astype(np.float32)
    spin = rng.uniform(-2.0, 2.0, 3).astype(np.float32)
    batch.vel += np.cross(spin, r).astype(np.float32)
    batch.vel[:, 2] -= np.float32(0.5)
    batch.vel += rng.random((n, 3), dtype=np.float32) * np.float32(0.1) - np.float32(0.05)
    f = rng.random((n, 9), dtype=np.float32) * np.float32(0.008) - np.float32(0.005)
    fluid = batch.model[:, 0] == 4
    f[fluid, 1:] = 0.0
    f[fluid, 4] = f[fluid, 8] = f[fluid, 0]
    batch.def_grad += f
    return batch


def _box_colliders():
    # a sticky floor: what lands on it stays in the scene however many passes follow
    return collider_array(box_walls(0.0, 1.0, BoundaryCondition.stick(), BoundaryCondition.slip()))


def _box(material, n, cells, seed, stream=0):
    """n uniformly random particles of one material in a box (8 to a cell where
    the sides' clamp to [0.1, 0.4] allows), above the floor of the unit box."""
    rng = np.random.default_rng([seed, stream])
    dx = 1.0 / cells
    shape = np.array([1.0, 0.8, 1.25])
    sides = np.clip(shape * (n * (dx / 2) ** 3) ** (1.0 / 3.0), 0.1, 0.4)
    lo = np.array([0.31, 0.27, 4.3 * dx])
    pos = (lo + sides * rng.random((n, 3))).astype(np.float32)
    density, model = _model(material)
    radius = np.float32(0.5 * (float(np.prod(sides)) / n) ** (1.0 / 3.0))
    batch = _in_motion(ParticleBatch.from_positions(pos, radius, density, model), rng)
    cols = _box_colliders()
    blocks = int(np.prod(np.ceil(sides / (4 * dx)) + 5))
    cap = 1
    while cap < 2 * blocks + 64:
        cap <<= 1
    return scenes.Scene("box", dx, 5.0e-5, (0.0, 0.0, -9.81), batch, cols, 0,
                        max(cap, scenes.grid_capacity_for(n)))


def _batch_sizes(case):
    r = random.Random(case["sizes"])
    return [_log_int(r, 4096, 131072) for _ in range(case["count"])]


def _coupled_sizes(case):
    return [_log_int(random.Random(2000 + s), 32768, 262144) for s in range(case["count"])]


def _scenes(case, seed):
    kind = case["kind"]
    if kind == "box":
        return [_box(case["material"], case["n"], case["cells"], seed)]
    if kind == "batch":
        return [_box("neo_hookean" if i % 2 else "sand", n, 128, seed, i) for i, n in enumerate(_batch_sizes(case))]
    if kind == "coupled":
        # bodies, mesh and placement are the scene's own (one set for all seeds); the sand moves with the seed
        got = []
        for s, n in enumerate(_coupled_sizes(case)):
            sc = scenes.coupled_scene(s, n_min=n, n_max=n)
            rng = np.random.default_rng([seed, s])
            sc.particles.pos += (rng.random((n, 3), dtype=np.float32) - np.float32(0.5)) * np.float32(0.5 * sc.dx)
            _in_motion(sc.particles, rng)
            got.append(sc)
        return got
    if kind == "cube":
        sc = scenes.elastic_cube(case["side"], seed=seed + 1)
        sc.colliders = _box_colliders()
    elif kind == "mixed":
        sc = scenes.mixed_materials(case["side"], seed=seed + 1)
    else:
        sc = scenes.sand_water(case["scale"], seed=seed + 1)
    _in_motion(sc.particles, np.random.default_rng(seed))
    return [sc]


def prepare(case, seed):
    scs = _scenes(case, seed)
    offsets = None
    if case["kind"] in ("batch", "coupled"):
        st, slots = batched_state_from_scenes(scs)
        offsets = batched_collider_offsets(scs, slots)
        if case.get("cpic"):
            st.set_use_cpic(True)
    else:
        st = state_from_scene(scs[0], deterministic=case.get("deterministic", False))
    n = sum(sc.n for sc in scs)
    state = {"case": case, "pipe": MpmPipeline(), "state": st, "n": n, "t": 0.0, "dt": scs[0].dt}
    if case["kind"] == "coupled":
        # what the program keeps to drive its bodies: their motions, not the particles
        state["bodies"] = ([scenes.Scene(sc.name, sc.dx, sc.dt, sc.gravity, None, sc.colliders, 0, 0,
                                         kinematics=sc.kinematics) for sc in scs], offsets)
    if case["out"] == "render":
        state["positions"] = torch.empty((n, 3), dtype=torch.float32, device="cuda")
        state["deformations"] = torch.empty((n, 9), dtype=torch.float32, device="cuda")
        state["colors"] = torch.empty((n, 4), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()  # the buffers are ready before the state's stream writes them
    return state


def run(state):
    case, pipe, st = state["case"], state["pipe"], state["state"]
    for _ in range(case["steps"]):
        if "bodies" in state:
            drive_kinematics(st, *state["bodies"], state["t"])
        pipe.step(st)
        state["t"] += state["dt"]
    if case["out"] == "read":
        return {"positions": st.read_positions(), "velocities": st.read_velocities()}
    st.prep_render(RENDER_VELOCITY, state["positions"].data_ptr(), state["deformations"].data_ptr(),
                   state["colors"].data_ptr())
    return {k: state[k] for k in ("positions", "deformations", "colors")}


# ---------------------------------------------------------------------------
# Work and tolerance
# ---------------------------------------------------------------------------

def _count(case):
    kind = case["kind"]
    if kind == "box":
        return case["n"]
    if kind == "cube":
        return case["side"] ** 3
    if kind == "mixed":
        return 6 * case["side"] ** 3
    if kind == "batch":
        return sum(_batch_sizes(case))
    if kind == "coupled":
        return sum(_coupled_sizes(case))
    s = [max(2, int(round(v * case["scale"]))) for v in (100, 100, 150, 50)]
    return s[0] * s[1] * (s[2] + s[3])


def work(case):
    """Per particle and step: position, velocity, affine matrix and deformation
    gradient read and written, mass, volume and material read (204 bytes), and
    24 more for the plastic models' words; 27 nodes to and from the grid.  Per
    frame: the outputs once."""
    n = _count(case)
    plastic = {"sand": 1.0, "sand_neo_hookean": 1.0, "snow": 1.0, "elastic": 0.0, "neo_hookean": 0.0, "water": 0.0}
    share = {"box": plastic.get(case.get("material"), 0.0), "cube": 0.0, "mixed": 0.5, "batch": 0.5,
             "column": 0.75, "coupled": 1.0}[case["kind"]]
    out = 64 if case["out"] == "render" else 24
    return {"bytes": n * (case["steps"] * (204 + 24 * share) + out), "flops": n * case["steps"] * 1000.0}


def tolerance(case):
    if case.get("deterministic"):
        return "exact"  # the mode's promise: the reference's order of operations, the same bits every time
    # 32-bit sums in another order, through a few substeps: two runs of the
    # same inputs (atomic order) differ by up to 8e-7, a run and the 64-bit
    # frame by up to 1.7e-6, or 1.2e-5 in the velocities of the mixed materials.
    return {"rel": 5e-5 if case["kind"] == "mixed" else 1e-5}


# ---------------------------------------------------------------------------
# The same frame in 64 bits
# ---------------------------------------------------------------------------

def _eigen(a):
    """Eigenvalues and vectors of symmetric 3x3 matrices (n, 3, 3), by Jacobi sweeps."""
    n = a.shape[0]
    d = {(i, j): a[:, i, j].clone() for i in range(3) for j in range(i, 3)}
    v = [[torch.full((n,), 1.0 if i == j else 0.0, dtype=a.dtype, device=a.device) for j in range(3)] for i in range(3)]
    for _ in range(6):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            apq = d[p, q]
            theta = (d[q, q] - d[p, p]) / (2.0 * torch.where(apq == 0, torch.ones_like(apq), apq))
            t = torch.where(theta >= 0, 1.0, -1.0) / (theta.abs() + torch.sqrt(1.0 + theta * theta))
            t = torch.where(apq == 0, torch.zeros_like(t), t)
            c = 1.0 / torch.sqrt(1.0 + t * t)
            s = t * c
            d[p, p], d[q, q] = d[p, p] - t * apq, d[q, q] + t * apq
            d[p, q] = torch.zeros_like(apq)
            r = 3 - p - q
            kp, kq = (min(p, r), max(p, r)), (min(q, r), max(q, r))
            d[kp], d[kq] = c * d[kp] - s * d[kq], s * d[kp] + c * d[kq]
            for i in range(3):
                v[i][p], v[i][q] = c * v[i][p] - s * v[i][q], s * v[i][p] + c * v[i][q]
    w = torch.stack([d[i, i] for i in range(3)], 1)
    return w, torch.stack([torch.stack(row, 1) for row in v], 1)


def _corotated(lam, mu, left, sig):
    """2 mu U (S - 1) S U^T + lambda (J - 1) J, with F V in `left`."""
    j = sig.prod(1)
    tau = torch.einsum("nik,nk,njk->nij", left, 2.0 * mu[:, None] * (sig - 1.0) / sig, left)
    return tau + (lam * (j - 1.0) * j)[:, None, None] * torch.eye(3, dtype=sig.dtype, device=sig.device)


def _neo_hookean(lam, mu, f):
    j = torch.linalg.det(f).clamp_min(1e-10)
    eye = torch.eye(3, dtype=f.dtype, device=f.device)
    return mu[:, None, None] * (f @ f.transpose(1, 2)) + (lam * torch.log(j) - mu)[:, None, None] * eye


def _stress(tag, w, st, f, grad):
    """Kirchhoff stress of particles of one model; f and the state words st are updated in place."""
    if tag == 1:
        return _neo_hookean(w[:, 0], w[:, 1], f)
    if tag == 4:
        j = torch.linalg.det(f).clamp_min(1e-6)
        sr = 0.5 * (grad + grad.transpose(1, 2))
        eye = torch.eye(3, dtype=f.dtype, device=f.device)
        dev = sr - (torch.einsum("nii->n", sr) / 3.0)[:, None, None] * eye
        p = torch.where(j <= 1.0, w[:, 0] * (j ** -w[:, 1] - 1.0), -w[:, 0] * w[:, 4] * (j - 1.0))
        return dev * (2.0 * w[:, 2] * j)[:, None, None] - (p * j)[:, None, None] * eye
    lam2, v = _eigen(f.transpose(1, 2) @ f)
    sig = lam2.clamp_min(1e-60).sqrt()
    left = f @ v
    if tag == 0:
        return _corotated(w[:, 0], w[:, 1], left, sig)
    if tag in (2, 3):
        ha, hb, hc, hd, plam, pmu, coh = (w[:, 3 + k] for k in range(7))
        q = st[:, 1]
        angle = torch.sin(ha + (hb * q - hd) * torch.exp(-hc * q))
        alpha = math.sqrt(2.0 / 3.0) * 2.0 * angle / (3.0 - angle)
        strain = torch.log(sig) + (st[:, 2] / 3.0)[:, None]
        tr = strain.sum(1)
        dev = strain - (tr / 3.0)[:, None]
        norm = dev.norm(dim=1)
        shifted = tr - coh
        tip = (shifted > 0.0) | (norm == 0.0)
        gamma = norm + (3.0 * plam + 2.0 * pmu) / (2.0 * pmu) * shifted * alpha
        inside = ~tip & (gamma <= 0.0)
        h = strain - dev * (gamma / norm.clamp_min(1e-300))[:, None]
        new = torch.where(tip[:, None], torch.exp(coh / 3.0)[:, None].expand_as(sig), torch.exp(h))
        hard = torch.where(tip, strain.norm(dim=1), gamma)
        keep = inside | (plam == 0.0)
        new = torch.where(keep[:, None], sig, new)
        d0, d1 = sig.prod(1), new.prod(1)
        st[:, 0] = torch.where(keep, st[:, 0], st[:, 0] * d0 / d1)
        st[:, 1] = torch.where(keep, st[:, 1], st[:, 1] + hard)
        st[:, 2] = torch.where(keep, st[:, 2], st[:, 2] + torch.log(d0) - torch.log(d1))
        left = left * (new / sig)[:, None, :]
        f.copy_(left @ v.transpose(1, 2))
        return _corotated(w[:, 10], w[:, 11], left, new) if tag == 2 else _neo_hookean(w[:, 10], w[:, 11], f)
    # snow
    new = torch.minimum(torch.maximum(sig, (1.0 - w[:, 1])[:, None]), (1.0 + w[:, 2])[:, None])
    st[:, 0] = (st[:, 0] * sig.prod(1) / new.prod(1)).clamp(0.1, 4.0)
    hard = torch.exp(w[:, 3] * (1.0 - st[:, 0]))
    left = left * (new / sig)[:, None, :]
    f.copy_(left @ v.transpose(1, 2))
    return _corotated(w[:, 4] * hard, w[:, 5] * hard, left, new)


def _walls(node, v, cols, dx, dt):
    """Projection of node velocities on resting, unrotated cuboids.  The
    geometry (which nodes lie within a cell of a wall) is that of 32-bit
    positions: a wall a whole number of cells away is a tie."""
    dist = torch.full((len(node),), math.inf, dtype=torch.float64, device=v.device)
    normal = torch.zeros_like(v)
    which = torch.full((len(node),), -1, dtype=torch.int64, device=v.device)
    x = node.float()
    half = torch.tensor(cols["shape_a"][:, :3].copy(), device=v.device)
    tra = torch.tensor(cols["translation"].copy(), device=v.device)
    cap = np.float32(1.5 * dx)
    for i in range(len(cols)):
        local = x - tra[i]
        lo, hi = -half[i] - local, local - half[i]
        shift = lo.clamp_min(0.0) - hi.clamp_min(0.0)
        outside = (shift != 0.0).any(1)
        # inside: out through the nearest face
        depth = torch.maximum(lo, hi)
        axis = depth.argmax(1, keepdim=True)
        sign = torch.where(lo.gather(1, axis) > hi.gather(1, axis), 1.0, -1.0)
        push = torch.zeros_like(shift).scatter_(1, axis, sign * depth.gather(1, axis))
        point = (local + torch.where(outside[:, None], shift, push)) + tra[i]
        d = point - x
        near = ~outside | (d.abs() <= float(cap)).all(1)
        length = d.double().norm(dim=1)
        sd = torch.where(outside, length, -length)
        better = near & (sd < dist)
        dist = torch.where(better, sd, dist)
        nv = d.double() / (length * torch.where(outside, -1.0, 1.0))[:, None]
        normal = torch.where(better[:, None], nv, normal)
        which = torch.where(better, torch.full_like(which, i), which)
    hit = which >= 0
    ty = torch.tensor(cols["bc_type"].astype(np.int64), device=v.device)[which.clamp_min(0)]
    fr = torch.tensor(cols["bc_friction"].astype(np.float64), device=v.device)[which.clamp_min(0)]
    vn = (v * normal).sum(1)
    tang = v - normal * vn[:, None]
    tl = tang.norm(dim=1)
    sep = torch.where((vn < 0.0)[:, None], tang * ((tl + fr * vn).clamp_min(0.0) / tl.clamp_min(1e-300))[:, None], v)
    inside = torch.where((ty == 0)[:, None], torch.zeros_like(v), torch.where((ty == 1)[:, None], tang,
                         torch.where((ty == 2)[:, None], sep, v)))
    far = v - normal * (vn + (dist - dx) / dt).clamp_max(0.0)[:, None]
    close = dist.float() <= np.float32(dx)
    return torch.where(hit[:, None], torch.where(close[:, None], inside, far), v)


def _frame(sc, steps):
    """`steps` substeps of one scene in 64 bits: positions, velocities, deformation gradients."""
    b, dev = sc.particles, "cuda" if torch.cuda.is_available() else "cpu"
    d = lambda a: torch.tensor(np.ascontiguousarray(a), device=dev).double()  # noqa: E731
    x, v, mass, vol, damp = d(b.pos), d(b.vel), d(b.mass), d(b.init_volume), d(b.damping)
    f = d(b.def_grad).reshape(-1, 3, 3).transpose(1, 2).contiguous()  # columns first
    c = d(b.aff).reshape(-1, 3, 3).transpose(1, 2).contiguous()
    tags = torch.tensor(b.model[:, 0].astype(np.int64), device=dev)
    w = d(b.model[:, 1:].copy().view(np.float32))
    groups = [(t, (tags == t).nonzero()[:, 0]) for t in range(6) if bool((tags == t).any())]
    st = w[:, :3].clone()
    dx, dt = float(np.float32(sc.dx)), float(np.float32(sc.dt))
    g = d(np.asarray(sc.gravity, np.float32))
    inv_d, lim = 4.0 / (dx * dx), dx / dt
    for _ in range(steps):
        cell = torch.sign(x) * torch.floor((x / dx).abs() + 0.5) - 1.0
        lo = cell.amin(0)
        dim = (cell.amax(0) - lo).long() + 3
        ref = cell * dx - x
        u = -ref / dx
        wt = (0.5 * (1.5 - u) ** 2, 0.75 - (u - 1.0) ** 2, 0.5 * (u - 0.5) ** 2)
        base = (cell - lo).long()
        base = (base[:, 0] * dim[1] + base[:, 1]) * dim[2] + base[:, 2]
        total = int(dim.prod())
        mom = torch.zeros((total, 4), dtype=torch.float64, device=dev)
        stencil = [(i, j, k, (i * dim[1] + j) * dim[2] + k) for i in range(3) for j in range(3) for k in range(3)]
        mv = v * mass[:, None]
        for i, j, k, off in stencil:
            s = torch.tensor([i, j, k], dtype=torch.float64, device=dev)
            weight = wt[i][:, 0] * wt[j][:, 1] * wt[k][:, 2]
            val = mv + torch.einsum("nij,nj->ni", c, ref + s * dx)
            mom.index_add_(0, base + off, torch.cat([val * weight[:, None], (mass * weight)[:, None]], 1))
        on = (mom[:, 3] > 0.0).nonzero()[:, 0]
        m = mom[on]
        nv = ((m[:, :3] + g * (m[:, 3:] * dt)) / m[:, 3:]).clamp(-lim, lim)
        idx = torch.stack([on // (dim[1] * dim[2]), (on // dim[2]) % dim[1], on % dim[2]], 1).double() + lo
        nv = _walls(idx * dx, nv, sc.colliders, dx, dt)
        grid = torch.zeros((total, 3), dtype=torch.float64, device=dev)
        grid[on] = nv
        v = torch.zeros_like(x)
        grad = torch.zeros_like(f)
        for i, j, k, off in stencil:
            s = torch.tensor([i, j, k], dtype=torch.float64, device=dev)
            wv = grid[base + off] * (wt[i][:, 0] * wt[j][:, 1] * wt[k][:, 2])[:, None]
            v += wv
            grad += wv[:, :, None] * (ref + s * dx)[:, None, :]
        grad *= inv_d
        speed = v.norm(dim=1)
        v = torch.where((speed > lim)[:, None], v / speed.clamp_min(1e-300)[:, None] * lim, v)
        v = v / (1.0 + damp * dt)[:, None]
        x = x + v * dt
        fluid = tags == 4
        rate = (torch.einsum("nii->n", grad) * dt / 3.0).clamp(-0.1, 0.1)
        size = (f[:, 0, 0] * (1.0 + rate)).clamp(0.5, 2.0)
        f = torch.where(fluid[:, None, None], size[:, None, None] * torch.eye(3, dtype=f.dtype, device=dev),
                        f + dt * grad @ f)
        tau = torch.zeros_like(f)
        for t, at in groups:
            ft, stt = f[at], st[at]
            tau[at] = _stress(t, w[at], stt, ft, grad[at])
            f[at], st[at] = ft, stt
        c = grad * mass[:, None, None] - tau * (vol * inv_d * dt)[:, None, None]
    return x, v, f.transpose(1, 2).reshape(-1, 9)


def exact(case, seed):
    if case["kind"] == "coupled":
        return None  # every node against 20k triangles a scene: minutes
    got = [(_frame(sc, case["steps"]), sc) for sc in _scenes(case, seed)]
    x, v, f = (torch.cat([p[k] for p, _ in got]) for k in range(3))
    if case["out"] == "read":
        return {"positions": x, "velocities": v}
    radius = torch.cat([torch.tensor(sc.particles.init_radius, device=x.device).double() for _, sc in got])
    color = torch.cat([v.abs() * (float(np.float32(got[0][1].dt)) * 100.0) + float(np.float32(0.2)),
                       torch.ones_like(v[:, :1])], 1)
    return {"positions": x, "deformations": f.clamp(-4.0, 4.0) * (2.0 * radius)[:, None], "colors": color}
