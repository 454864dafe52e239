"""Performance cases of the cell-grid Lennard-Jones path: what a program that uses `ljcell` has it do.

A case is a dict of plain values.  `prepare` makes what such a program holds before the call (inputs
on the GPU, or in pinned host memory for the host-buffer entry, its output buffers, and the plan of
a batch), `run` makes one pass through the public entry points and returns its whole outputs, `exact`
restates the outputs that are computed numbers in 64-bit torch without the library, and `work` counts
the bytes and flops that a pass cannot do without.

Kinds of case, by the call a program makes:
  step     bin + compute of a uniform box (both within-cell orders)
  shell    bin + compute of particles on a sphere surface in a mostly empty grid
  verlet   one velocity-Verlet step of a dense fluid, from a state the program keeps
  law      bin + the reference's law (energies over the whole 27-cell stencil)
  mixed    bin + mixed-precision records + the mixed-precision law
  batch    many uneven systems as one graph replay
  cells    the cell list alone: point3d input, every optional output, the candidate count
  host     one step from and to the program's own host buffers
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "particle-interaction-with-optix_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

import ljcell  # noqa: E402

DEVICE = "cuda"
UNIT = ((0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
SHELL_BOX = ((-0.5, -0.5, -0.5), (1.5, 1.5, 1.5))
LATTICE_DT, LATTICE_MASS = 2e-4, 1.0
ORDERS = {"x": ljcell.ORDER_X, "index": ljcell.ORDER_INDEX}


def listed():
    return [
        # the smallest systems a program steps: a test fluid, every launch and call counts
        {"name": "step_1k", "kind": "step", "n": 1000, "cutoff": 0.25, "order": "x"},
        # the small reference configuration: 100,000 particles, about 52 neighbours each
        {"name": "step_100k", "kind": "step", "n": 100_000, "cutoff": 0.05, "order": "x"},
        # the headline configuration: 10 million particles, about 42 neighbours each
        {"name": "step_10M", "kind": "step", "n": 10_000_000, "cutoff": 0.01, "order": "x"},
        # the dense configuration: about 335 neighbours each, all arithmetic
        {"name": "dense_10M", "kind": "step", "n": 10_000_000, "cutoff": 0.02, "order": "x"},
        # a caller that needs the stable (input-index) order inside each cell; a ragged size
        {"name": "stable_1M", "kind": "step", "n": 1_000_003, "cutoff": 0.0217, "order": "index"},
        # the sparse configuration: a sphere surface, 64 million cells of which 1% are occupied
        {"name": "shell_4M", "kind": "shell", "n": 4_000_000, "cutoff": 0.005},
        # time stepping of a fluid near its equilibrium density, a ragged lattice of 119^3
        {"name": "verlet_1.7M", "kind": "verlet", "side": 119},
        # the reference's own law at one of its sweep's densities (64 divisions, 16 per cell)
        {"name": "law_4M", "kind": "law", "n": 4_194_304, "cutoff": 1.0 / 64.0},
        # the mixed-precision form where it is meant to be used, in the dense regime
        {"name": "mixed_2M", "kind": "mixed", "n": 2_000_003, "cutoff": 0.0345},
        # uneven systems (1,000 to 200,000 particles, 20 to 200 neighbours, a quarter of them shells)
        {"name": "batch_128", "kind": "batch", "systems": 128, "shapes": 1234},
        # another program's neighbour search: the cell list with all its views
        {"name": "cells_3M", "kind": "cells", "n": 3_000_017, "cutoff": 0.0167},
        # a program whose particles live in host memory: copies in and out count
        {"name": "host_1M", "kind": "host", "n": 1_000_000, "cutoff": 0.0215},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, n_lo, n_hi, cell_lo, cell_hi):
    """Particles and cutoff of a unit box: n and the particles per cell spread over their logarithm."""
    n = int(round(_log(rng, n_lo, n_hi)))
    per_cell = _log(rng, cell_lo, cell_hi)
    return n, min(1.0 / 3.0, (per_cell / n) ** (1.0 / 3.0))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "stable", "shell", "verlet", "law", "mixed", "batch", "cells", "host"])
    if kind in ("step", "stable"):
        n, rc = _box(rng, 1000, 10_000_000, 0.5, 80.0) if kind == "step" else _box(rng, 1000, 4_000_000, 1.0, 32.0)
        return {"kind": "step", "n": n, "cutoff": rc, "order": "x" if kind == "step" else "index"}
    if kind == "shell":
        n = int(round(_log(rng, 50_000, 4_000_000)))
        return {"kind": "shell", "n": n, "cutoff": max(0.005, 2.0 * math.sqrt(rng.uniform(20.0, 60.0) / n))}
    if kind == "verlet":
        return {"kind": "verlet", "side": int(round(_log(rng, 15.0, 150.0)))}
    if kind == "law":
        n, rc = _box(rng, 10_000, 4_200_000, 4.0, 32.0)
        return {"kind": "law", "n": n, "cutoff": rc}
    if kind == "mixed":
        n, rc = _box(rng, 50_000, 2_000_000, 10.0, 80.0)
        return {"kind": "mixed", "n": n, "cutoff": rc}
    if kind == "batch":
        return {"kind": "batch", "systems": rng.randint(16, 128), "shapes": rng.randint(1, 1_000_000)}
    if kind == "cells":
        n, rc = _box(rng, 20_000, 4_000_000, 1.0, 32.0)
        return {"kind": "cells", "n": n, "cutoff": rc}
    n, rc = _box(rng, 10_000, 2_000_000, 5.0, 40.0)
    return {"kind": "host", "n": n, "cutoff": rc}


# ------------------------------------------------------------------ what a program holds
_CONTEXT = []


def _context():
    """The one handle that a program keeps for all its systems."""
    if not _CONTEXT:
        _CONTEXT.append(ljcell.Context(0))
    return _CONTEXT[0]


def _bounds(case):
    return SHELL_BOX if case["kind"] == "shell" else UNIT


def _uniform(n, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    return [torch.rand(n, dtype=torch.float32, device=DEVICE, generator=gen) for _ in range(3)]


def _sphere(n, seed):
    """Points on the unit sphere about (0.5, 0.5, 0.5): theta = 2 pi u, phi = acos(1 - 2 u)."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    u = torch.rand((2, n), dtype=torch.float64, device=DEVICE, generator=gen)
    theta, c = 2.0 * math.pi * u[0], 1.0 - 2.0 * u[1]
    s = torch.sqrt(torch.clamp(1.0 - c * c, min=0.0))
    return [(0.5 + v).to(torch.float32) for v in (s * torch.cos(theta), s * torch.sin(theta), c)]


def _positions(case, seed):
    return _sphere(case["n"], seed) if case["kind"] == "shell" else _uniform(case["n"], seed)


def _lattice(side, seed):
    """A jittered cubic lattice in sorted order of no grid: positions, velocities and the restoring
    forces of the jitter (the forces a program holds from its last step), all float32."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    a = 1.0 / side
    axis = (torch.arange(side, dtype=torch.float64, device=DEVICE) + 0.5) * a
    site = torch.stack(torch.meshgrid(axis, axis, axis, indexing="ij"), dim=-1).reshape(-1, 3)
    n = site.shape[0]
    u = (torch.rand((n, 3), dtype=torch.float64, device=DEVICE, generator=gen) - 0.5) * (0.1 * a)
    vel = torch.randn((n, 3), dtype=torch.float32, device=DEVICE, generator=gen) * 0.5
    sigma = a / 1.12
    return (site + u).to(torch.float32), vel, (u * (-150.0 / sigma ** 2)).to(torch.float32)


def _lattice_law(side):
    sigma = 1.0 / side / 1.12
    return 2.5 * sigma, sigma


def _systems(case):
    return ljcell.batch_workload(nsys=case["systems"], seed=case["shapes"])


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx}
    if kind == "batch":
        systems = _systems(case)
        parts = [_sphere(d["n"], seed * 4096 + i) if d["kind"] == "shell" else _uniform(d["n"], seed * 4096 + i)
                 for i, d in enumerate(systems)]
        s["batch"] = ljcell.Batch(ctx, systems)
        s["xyz"] = [torch.cat([q[k] for q in parts]) for k in range(3)]
        s["out"] = s["batch"].alloc_outputs()
        return s
    if kind == "verlet":
        rc, sigma = _lattice_law(case["side"])
        pos, vel, force = _lattice(case["side"], seed)
        s["grid"], s["params"] = ljcell.grid_from_box(*UNIT, rc), ljcell.params(rc, sigma=sigma)
        b = ctx.bin(s["grid"], *[pos[:, k].contiguous() for k in range(3)])
        ids = b.xyzi[:, 3].contiguous().view(torch.int32).long()
        s["binned"], s["kept"] = b, (b.xyzi.clone(), vel[ids].contiguous(), force[ids].contiguous())
        s["vel"], s["force"] = torch.empty_like(vel), torch.empty_like(force)
        s["energy"] = torch.empty(b.n, dtype=torch.float32, device=DEVICE)
        s["totals"] = torch.zeros(4, dtype=torch.float64, device=DEVICE)
        return s
    n, rc = case["n"], case["cutoff"]
    s["grid"], s["params"] = ljcell.grid_from_box(*_bounds(case), rc), ljcell.params(rc)
    xyz = _positions(case, seed)
    if kind == "host":
        pinned = [torch.empty(n, dtype=torch.float32, pin_memory=True) for _ in range(3)]
        for h, v in zip(pinned, xyz):
            h.copy_(v)
        s["keep"] = pinned + [torch.empty(n, dtype=torch.float32, pin_memory=True),
                              torch.empty((n, 3), dtype=torch.float32, pin_memory=True)]
        s["xyz"], s["energy"], s["force"] = [h.numpy() for h in pinned], s["keep"][3].numpy(), s["keep"][4].numpy()
        return s
    if kind == "cells":
        s["points"] = torch.stack(xyz, dim=1).reshape(-1)
        s["binned"] = ctx.alloc_binned(s["grid"], n, ljcell.ORDER_X, soa=True, cells=True)
        s["candidates"] = torch.empty(1, dtype=torch.int64, device=DEVICE)
        return s
    s["xyz"], s["order"] = xyz, ORDERS[case.get("order", "x")]
    s["binned"] = ctx.alloc_binned(s["grid"], n, s["order"])
    s["energy"], s["force"], s["totals"] = ctx.alloc_outputs(n)
    if kind == "mixed":
        s["rec"] = torch.empty((n, 2), dtype=torch.float32, device=DEVICE)
    return s


# ------------------------------------------------------------------ one pass
def _totals(t):
    """Energy and virial in float32, and the pair count as the integer that it is."""
    t = t.reshape(-1, 4)
    return {"energy_virial": t[:, :2].to(torch.float32), "pairs": t.view(torch.int64)[:, 2]}


def _cell_grid(b):
    return {"counts": b.counts, "offsets": b.offsets, "cell": b.cell, "xyzi": b.xyzi}


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind == "batch":
        energy, force, index, totals = state["out"]
        state["batch"].run(*state["xyz"], energy, force, index, totals, mode="graph")
        return {"energy": energy, "force": force, "index": index, "totals": _totals(totals)}
    g = state["grid"]
    if kind == "host":
        t = ctx.simulate_host_inorder(g, state["params"], *state["xyz"], state["energy"], state["force"])
        return {"energy": state["energy"], "force": state["force"], "total_energy": t.energy, "virial": t.virial,
                "pairs": t.pairs}
    if kind == "cells":
        p, b = state["points"], state["binned"]
        ctx.bin(g, p, p[1:], p[2:], stride=3, out=b)
        ctx.count_candidates(g, b.offsets, state["candidates"])
        return {**_cell_grid(b), "cells": b.cells, "x": b.sx, "y": b.sy, "z": b.sz, "index": b.index,
                "candidates": state["candidates"]}
    if kind == "verlet":
        # a trial step from the state that the program keeps (and returns to when it rejects the step)
        b = state["binned"]
        for to, kept in zip((b.xyzi, state["vel"], state["force"]), state["kept"]):
            to.copy_(kept)
        ctx.step_verlet(g, state["params"], b, state["vel"], state["force"], LATTICE_DT, LATTICE_MASS, state["energy"],
                        state["totals"])
        return {**_cell_grid(b), "vel": state["vel"], "force": state["force"], "energy": state["energy"],
                "totals": _totals(state["totals"])}
    b = ctx.bin(g, *state["xyz"], order=state["order"], out=state["binned"])
    if kind == "law":
        return {**_cell_grid(b), "energy": ctx.compute_compat(g, b, state["energy"])}
    if kind == "mixed":
        ctx.pack_mixed(g, b, state["rec"])
        ctx.compute_mixed(g, state["params"], b, state["rec"], state["energy"], state["force"], state["totals"])
        return {**_cell_grid(b), "rec": state["rec"], "energy": state["energy"], "force": state["force"],
                "totals": _totals(state["totals"])}
    ctx.compute(g, state["params"], b, state["energy"], state["force"], state["totals"])
    return {**_cell_grid(b), "energy": state["energy"], "force": state["force"], "totals": _totals(state["totals"])}


# ------------------------------------------------------------------ work
def _grid_dims(lo, hi, rc):
    f = np.float32
    return [max(1, int((f(h) - f(a)) / f(rc))) for a, h in zip(lo, hi)]


def _law_work(n, neighbours, ncells, out_bytes, pair_flops=26.0):
    """Positions in, counts and offsets, sorted records with their cells, and the outputs; a distance
    (8 flops) and the law (18) per interacting pair."""
    return {"bytes": n * (12.0 + 20.0 + out_bytes) + 8.0 * ncells, "flops": n * neighbours * pair_flops}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for d in _systems(case):
            w = _law_work(d["n"], d["neighbours"], math.prod(_grid_dims(d["lo"], d["hi"], d["cutoff"])), 20.0)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "verlet":
        n, (rc, _) = case["side"] ** 3, _lattice_law(case["side"])
        w = _law_work(n, 4.0 / 3.0 * math.pi * rc ** 3 * n, math.prod(_grid_dims(*UNIT, rc)), 16.0)
        return {"bytes": w["bytes"] + n * (4.0 + 12.0 + 12.0 + 12.0), "flops": w["flops"] + 18.0 * n}
    n, rc = case["n"], case["cutoff"]
    ncells = math.prod(_grid_dims(*_bounds(case), rc))
    if kind == "cells":
        return {"bytes": n * (12.0 + 20.0 + 16.0) + 16.0 * ncells, "flops": 10.0 * n}
    if kind == "law":
        return _law_work(n, 27.0 * n / ncells, ncells, 4.0, pair_flops=18.0)
    if kind == "shell":
        return _law_work(n, n * rc * rc / 4.0, ncells, 16.0)
    neighbours = 4.0 / 3.0 * math.pi * rc ** 3 * n
    if kind == "mixed":
        return _law_work(n, neighbours, ncells, 24.0)
    if kind == "host":
        return {"bytes": n * (12.0 + 16.0), "flops": n * neighbours * 26.0}
    return _law_work(n, neighbours, ncells, 16.0)


# ------------------------------------------------------------------ 64-bit restatement
def _scalar(v, dtype):
    return torch.tensor(float(v), dtype=dtype, device=DEVICE)


def _sorted_system(xyz, lo, hi, rc, order):
    """Cell-sorted particles as plain torch has them: permutation, cell coordinates, offsets, dims."""
    dims = _grid_dims(lo, hi, rc)
    w = _scalar(np.float32(rc), torch.float32)
    c = []
    for k in range(3):
        q = ((xyz[k] - _scalar(np.float32(lo[k]), torch.float32)) / w).clamp(0, dims[k])
        c.append(q.to(torch.int64).clamp(max=dims[k] - 1))
    cell = (c[2] * dims[1] + c[1]) * dims[0] + c[0]
    perm = torch.argsort(xyz[0], stable=True) if order == "x" else torch.arange(len(cell), device=DEVICE)
    perm = perm[torch.argsort(cell[perm], stable=True)]
    counts = torch.bincount(cell, minlength=math.prod(dims))
    off = torch.zeros(math.prod(dims) + 1, dtype=torch.int64, device=DEVICE)
    torch.cumsum(counts, 0, out=off[1:])
    return perm, [v[perm] for v in c], off, dims


def _rows(c, off, dims, base=0):
    """The 9 stencil rows of every particle: (dy, dz, first, end) of the sorted particles in each."""
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            z, y = c[2] + dz, c[1] + dy
            ok = (z >= 0) & (z < dims[2]) & (y >= 0) & (y < dims[1])
            r = (z.clamp(0, dims[2] - 1) * dims[1] + y.clamp(0, dims[1] - 1)) * dims[0]
            s = off[r + (c[0] - 1).clamp(min=0)]
            e = torch.where(ok, off[r + (c[0] + 1).clamp(max=dims[0] - 1) + 1], s)
            yield dy, dz, s + base, e + base


def _add_law(sums, k, j, ok, d, hit, sig2):
    """Adds the truncated law of candidates j on targets k; d the 64-bit differences."""
    hit = hit & ok & (j != k)
    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    s2 = torch.where(hit, sig2 / r2, 0.0)
    s6 = s2 * s2 * s2
    s12 = s6 * s6
    t = 2.0 * s12 - s6
    sums[0] += s12 - s6
    sums[1] += t
    for q in range(3):
        sums[2 + q] -= torch.where(hit, t * s2 * d[q], 0.0)


def _truncated(p, rows, rc, sigma, mixed_uyz=None, width=None, chunk=4_000_000):
    """Energy (n), force (n, 3) and (total energy, virial) of the truncated law (eps = 1) in 64 bits.
    p: sorted float32 positions; rows: (dy, dz, first, end) per stencil row; rc, sigma: float32
    numbers or one per particle.  With mixed_uyz the stored positions are (x, uy, uz) in cell units."""
    n = len(p[0])
    rc2 = rc * rc
    outs = [torch.zeros(n, dtype=torch.float64, device=DEVICE) for _ in range(5)]
    every = torch.arange(n, device=DEVICE)
    sig2 = sigma.double() ** 2
    for a in range(0, n, chunk):
        z = slice(a, min(n, a + chunk))
        k = every[z]
        sums = [torch.zeros(len(k), dtype=torch.float64, device=DEVICE) for _ in range(5)]
        pk = [v[z] for v in p]
        for dy, dz, first, end in rows:
            first, end = first[z], end[z]
            for t in range(int((end - first).max()) if len(k) else 0):
                j = (first + t).clamp(max=n - 1)
                ok = first + t < end
                if mixed_uyz is None:
                    f = [v[j] - q for v, q in zip(p, pk)]           # the float distance test
                    d = [v.double() for v in f]
                    r2 = ((d[2] * d[2] + (d[1] * d[1] + (f[0] * f[0]).double()).float().double())).float()
                    hit = r2 < (rc2 if rc2.ndim == 0 else rc2[z])
                    d = [v[j].double() - q.double() for v, q in zip(p, pk)]
                    _add_law(sums, k, j, ok, d, hit, sig2 if sig2.ndim == 0 else sig2[z])
                else:
                    w = width.double()
                    d = [p[0][j].double() - pk[0].double()]
                    d += [(u[j].double() - u[z].double() + o) * w for u, o in zip(mixed_uyz, (dy, dz))]
                    hit = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] < rc2.double()
                    _add_law(sums, k, j, ok, d, hit, sig2)
        for o, v in zip(outs, sums):
            o[z] = v
    force = torch.stack([v * (24.0 / sig2) for v in outs[2:]], dim=1)
    return 4.0 * outs[0], force, outs[0], outs[1]


def _energy_virial(e, w):
    return {"energy_virial": torch.stack([2.0 * e.sum(), 12.0 * w.sum()]).reshape(1, 2), "pairs": None}


def _reference_law(p, rows, chunk=4_000_000):
    """The reference's law: 4 (r^-12 - r^-6), r^2 = d.d + 1e-5, over the whole stencil."""
    n = len(p[0])
    v = torch.zeros(n, dtype=torch.float64, device=DEVICE)
    every = torch.arange(n, device=DEVICE)
    for a in range(0, n, chunk):
        z = slice(a, min(n, a + chunk))
        pk = [q[z].double() for q in p]
        for _, _, first, end in rows:
            first, end = first[z], end[z]
            for t in range(int((end - first).max())):
                j = (first + t).clamp(max=n - 1)
                ok = (first + t < end) & (j != every[z])
                r2 = 1e-5
                for q, b in zip(p, pk):
                    r2 = r2 + (q[j].double() - b) ** 2
                r6 = 1.0 / (r2 * r2 * r2)
                v[z] += torch.where(ok, r6 * r6 - r6, 0.0)
    return 4.0 * v


_NO_GRID = {"counts": None, "offsets": None, "cell": None, "xyzi": None}


def _exact_batch(case, seed):
    """All systems at once: their rows hold indices into the concatenated sorted particles."""
    systems = _systems(case)
    parts, rows, rcs, sigmas = [], [[] for _ in range(9)], [], []
    base = 0
    for i, d in enumerate(systems):
        xyz = _sphere(d["n"], seed * 4096 + i) if d["kind"] == "shell" else _uniform(d["n"], seed * 4096 + i)
        perm, c, off, dims = _sorted_system(xyz, d["lo"], d["hi"], d["cutoff"], "x")
        parts.append([v[perm] for v in xyz])
        for r, row in enumerate(_rows(c, off, dims, base)):
            rows[r].append(row)
        rc = np.float32(d["cutoff"])
        rcs.append(torch.full((d["n"],), float(rc), dtype=torch.float32, device=DEVICE))
        sigmas.append(torch.full((d["n"],), float(rc / np.float32(2.5)), dtype=torch.float32, device=DEVICE))
        base += d["n"]
    p = [torch.cat([q[k] for q in parts]) for k in range(3)]
    joined = [(r[0][0], r[0][1], torch.cat([q[2] for q in r]), torch.cat([q[3] for q in r])) for r in rows]
    energy, force, e, w = _truncated(p, joined, torch.cat(rcs), torch.cat(sigmas))
    split = [d["n"] for d in systems]
    ev = torch.stack([torch.stack([2.0 * a.sum(), 12.0 * b.sum()]) for a, b in zip(e.split(split), w.split(split))])
    return {"energy": energy, "force": force, "index": None, "totals": {"energy_virial": ev, "pairs": None}}


def exact(case, seed):
    kind = case["kind"]
    if kind == "cells":
        return None
    if kind == "batch":
        return _exact_batch(case, seed)
    f32 = torch.float32
    if kind == "verlet":
        rc, sigma = (np.float32(v) for v in _lattice_law(case["side"]))
        pos, vel, force = _lattice(case["side"], seed)
        # the kept state is in the sorted order of the positions before the step
        first = _sorted_system([pos[:, k].contiguous() for k in range(3)], *UNIT, rc, "x")[0]
        pos, vel, force = pos[first], vel[first], force[first]
        h = _scalar(np.float32(0.5) * np.float32(LATTICE_DT) / np.float32(LATTICE_MASS), f32)
        half = vel + h * force
        moved = pos + _scalar(np.float32(LATTICE_DT), f32) * half
        xyz = [moved[:, k].contiguous() for k in range(3)]
        perm, c, off, dims = _sorted_system(xyz, *UNIT, rc, "x")
        energy, force, e, w = _truncated([v[perm] for v in xyz], list(_rows(c, off, dims)), _scalar(rc, f32),
                                         _scalar(sigma, f32))
        return {**_NO_GRID, "vel": half[perm].double() + h.double() * force, "force": force, "energy": energy,
                "totals": _energy_virial(e, w)}
    rc = np.float32(case["cutoff"])
    xyz = _positions(case, seed)
    lo, hi = _bounds(case)
    perm, c, off, dims = _sorted_system(xyz, lo, hi, rc, case.get("order", "x"))
    p = [v[perm] for v in xyz]
    rows = list(_rows(c, off, dims))
    if kind == "law":
        return {**_NO_GRID, "energy": _reference_law(p, rows)}
    sigma = _scalar(rc / np.float32(2.5), f32)
    rc = _scalar(rc, f32)
    if kind == "mixed":
        uyz = []
        for q, cell in ((p[1], c[1]), (p[2], c[2])):
            origin = (cell.double() * rc.double()).to(f32)
            uyz.append(((q - origin) / rc).to(torch.float16))
        energy, force, e, w = _truncated(p, rows, rc, sigma, mixed_uyz=uyz, width=rc)
        return {**_NO_GRID, "rec": None, "energy": energy, "force": force, "totals": _energy_virial(e, w)}
    energy, force, e, w = _truncated(p, rows, rc, sigma)
    if kind == "host":
        back = torch.empty_like(perm)
        back[perm] = torch.arange(len(perm), device=DEVICE)
        return {"energy": energy[back], "force": force[back], "total_energy": 2.0 * float(e.sum()),
                "virial": 12.0 * float(w.sum()), "pairs": None}
    return {**_NO_GRID, "energy": energy, "force": force, "totals": _energy_virial(e, w)}
