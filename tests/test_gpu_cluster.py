"""The cluster walk (pair kernel 1) at the edges of its tiles: clusters of 8 and groups of 16 targets
filled to every remainder, segments of 16 cells, candidate lists that overflow and are walked in parts,
and target ranges that cut groups; both within-cell orders, against the FP64 oracle with the tolerances
of test_gpu_parity."""
import numpy as np
import pytest

import ljoracle as O
from test_gpu_parity import ENERGY_SCALED_TOL, FORCE_NORMWISE_TOL, FORCE_SCALED_TOL, dev, np_

pytestmark = pytest.mark.gpu

# name: box, cell width, cutoff, particles
SHAPES = {
    **{f"one_cell_{n}": (((0, 0, 0), (1, 1, 1)), 1.0, 1.0, n) for n in (1, 7, 8, 9, 15, 16, 17, 31, 33)},
    "row_of_33_cells": (((0, 0, 0), (3.3, 0.1, 0.1)), 0.1, 0.1, 800),        # three segments, the last one cell long
    "list_overflows": (((0, 0, 0), (0.3, 0.3, 0.3)), 0.1, 0.1, 9000),        # about 1,400 candidates per list
    "thin_rows": (((0, 0, 0), (4.0, 1.0, 1.0)), 0.1, 0.1, 3000),             # under one particle per cell
    "cutoff_below_width": (((-1, 2, 5), (1, 3, 6)), 0.125, 0.06, 20000),
}


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("name", list(SHAPES))
def test_cluster_walk_edges(torch_cuda, ctx, name, order):
    import ljcell

    torch = torch_cuda
    (lo, hi), width, rc, n = SHAPES[name]
    rng = np.random.default_rng(n + order)
    lo32, hi32 = np.array(lo, np.float32), np.array(hi, np.float32)
    pts = (lo32 + (hi32 - lo32) * rng.random((n, 3), dtype=np.float32)).astype(np.float32)
    x, y, z = (np.ascontiguousarray(pts[:, k]) for k in range(3))
    g, og = ljcell.grid_from_box(lo, hi, width), O.grid_from_box(lo, hi, width)
    p = ljcell.params(rc, sigma=rc / 10)   # few close pairs: energies stay in the float range
    ctx.set_tuning(1)
    try:
        b = ctx.bin(g, dev(torch, x), dev(torch, y), dev(torch, z), order=order)
        e, f, tot = ctx.compute(g, p, b)
        parts = []
        for kb, ke in ((0, n // 3), (n // 3, n // 3 + 5), (n // 3 + 5, n)):
            kb, ke = min(kb, n), min(max(ke, kb), n)
            pe, pf, pt = ctx.alloc_outputs(n)
            pe.fill_(float("nan"))
            ctx.compute_range(g, p, b, kb, ke, pe, pf, pt)
            parts.append((kb, ke, pe, pf, pt))
        ctx.sync()
    finally:
        ctx.set_tuning(0)
    ob = O.bin_particles(og, x, y, z, order)
    ref = O.config_forces(og, ob, rc, 1.0, p.sigma)
    t = ljcell.totals_from_tensor(tot)
    assert t["pairs"] == ref.pairs
    fe, ee = ref.force_errors(np_(f)[:n], FORCE_SCALED_TOL), ref.energy_errors(np_(e)[:n], ENERGY_SCALED_TOL)
    assert fe["max_scaled_over_tol"] <= 1.0 and ee["max_scaled_over_tol"] <= 1.0
    if ref.pairs:
        assert fe["normwise"] <= FORCE_NORMWISE_TOL
    # a range of targets: their bits, nothing outside the range, and pair counts that add up
    assert sum(ljcell.totals_from_tensor(q[4])["pairs"] for q in parts) == ref.pairs
    for kb, ke, pe, pf, _ in parts:
        assert torch.equal(pe[kb:ke].view(torch.int32), e[kb:ke].view(torch.int32))
        assert torch.equal(pf[kb:ke].view(torch.int32), f[kb:ke].view(torch.int32))
        assert bool(torch.isnan(pe[:kb]).all()) and bool(torch.isnan(pe[ke:n]).all())


@pytest.mark.parametrize("name", [f"one_cell_{n}" for n in (8, 9, 15, 16, 17, 31, 33)] + ["row_of_33_cells", "list_overflows",
                                                                                          "cutoff_below_width"])
def test_mixed_cluster_walk_edges(torch_cuda, ctx, name):
    """The mixed form's cluster walk at the same edges, against FP64 on the stored positions."""
    import ljcell

    torch = torch_cuda
    (lo, hi), width, rc, n = SHAPES[name]
    rng = np.random.default_rng(n)
    lo32, hi32 = np.array(lo, np.float32), np.array(hi, np.float32)
    pts = (lo32 + (hi32 - lo32) * rng.random((n, 3), dtype=np.float32)).astype(np.float32)
    x, y, z = (np.ascontiguousarray(pts[:, k]) for k in range(3))
    g, og = ljcell.grid_from_box(lo, hi, width), O.grid_from_box(lo, hi, width)
    assert n >= 8 * g.ncells
    p = ljcell.params(rc, sigma=rc / 10)
    b = ctx.bin(g, dev(torch, x), dev(torch, y), dev(torch, z))
    e, f, tot = ctx.compute_mixed(g, p, b, ctx.pack_mixed(g, b))
    ctx.sync()
    ob = O.bin_particles(og, x, y, z, O.ORDER_X)
    ref = O.mixed_forces(og, ob, *O.pack_mixed(og, ob), rc, 1.0, p.sigma)
    assert ljcell.totals_from_tensor(tot)["pairs"] == ref.pairs
    fe, ee = ref.force_errors(np_(f)[:n]), ref.energy_errors(np_(e)[:n])
    assert fe["max_scaled"] <= FORCE_SCALED_TOL and fe["normwise"] <= FORCE_NORMWISE_TOL
    assert ee["max_scaled"] <= ENERGY_SCALED_TOL


def test_batch_walk_chosen_by_occupied_cells(torch_cuda, ctx):
    """Batched systems of 2 to 6 particles per cell of their whole grid take the cluster walk or the
    two-target walk by the occupancy of the cells that hold particles, decided on the device: uniform and
    shell systems, an empty and a one-particle one; the batched step, its graph replay and the per-system
    launches agree bit for bit, and every pair count with lj_compute's."""
    import ljcell

    torch = torch_cuda
    unit, box = ((0, 0, 0), (1, 1, 1)), ((-0.5,) * 3, (1.5,) * 3)
    systems = []
    for i, (kind, n, rc) in enumerate([("uniform", 3000, 0.1), ("shell", 20000, 0.11), ("uniform", 0, 0.1),
                                       ("uniform", 5001, 0.1), ("shell", 9000, 0.15), ("uniform", 1, 0.3)]):
        lo, hi = unit if kind == "uniform" else box
        systems.append({"kind": kind, "n": n, "cutoff": rc, "lo": lo, "hi": hi, "seed": 40 + i})
    b = ljcell.Batch(ctx, systems)
    per_cell = [d["n"] / b.grid(s).ncells for s, d in enumerate(systems)]
    assert all(2 <= per_cell[s] < 6 for s in (0, 1, 3, 4))
    xyz = b.generate()
    outs = []
    for mode in ("plain", "separate", "graph", "graph"):
        e, f, idx, tot = b.alloc_outputs()
        b.run(*xyz, e, f, idx, tot, mode=mode)
        ctx.sync()
        outs.append((np_(e), np_(f), np_(idx), ljcell.totals_from_array(tot)))
    for o in outs[1:]:
        for x, y in zip(outs[0][:3], o[:3]):
            assert np.array_equal(x.view(np.uint8), y.view(np.uint8))
        assert [t["pairs"] for t in o[3]] == [t["pairs"] for t in outs[0][3]]
    for s, d in enumerate(systems):
        sl = slice(d["first"], d["first"] + d["n"])
        g = b.grid(s)
        q = ctx.bin(g, *(t[sl].contiguous() for t in xyz))
        _, _, tot = ctx.compute(g, b.params(s), q)
        ctx.sync()
        assert ljcell.totals_from_tensor(tot)["pairs"] == outs[0][3][s]["pairs"], s
    b.close()
