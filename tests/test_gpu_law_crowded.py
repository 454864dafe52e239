"""The reference law's warp-per-cell kernel where cells hold many more targets than one warp should take: few
cells, droplets in a filled grid, and cells at the edges of its chunks (16 targets on few cells, 64 on grids
that fill the GPU); against the law in 64 bits within the reference's own tolerance (the float oracle adds a target's
terms one after the other and is itself off by up to 3e-5 on the droplets).  A cell id outside the grid is
reported by both kernels of the law."""
import numpy as np
import pytest

import ljoracle as O
from test_gpu_parity import COMPAT_REL_TOL, dev, np_

pytestmark = pytest.mark.gpu


def uniform(n, seed):
    return np.random.default_rng(seed).random((n, 3), dtype=np.float32)


def droplet(n, rc, share, seed):
    """A share of the particles in one cell of the grid."""
    p = uniform(n, seed)
    k = int(n * share)
    p[:k] = (np.floor(0.5 / rc) + 0.01 + 0.98 * p[:k]).astype(np.float32) * np.float32(rc)
    return p.astype(np.float32)


def cells_of(counts, side, seed):
    """counts[i] particles in cell i of side^3 unit-box cells."""
    rng = np.random.default_rng(seed)
    c = np.repeat(np.arange(len(counts)), counts)
    ijk = np.stack([c % side, c // side % side, c // side ** 2], 1)
    return ((ijk + 0.01 + 0.98 * rng.random((len(c), 3))) / side).astype(np.float32)


def law64(og, ob):
    """The law in 64 bits, cell by cell, over the oracle's binned particles."""
    p, off = np.stack([ob.sx, ob.sy, ob.sz], 1).astype(np.float64), ob.offsets
    gx, gy, gz = og.dim
    v = np.zeros(len(p))
    for c in np.unique(ob.cell_sorted):
        x, y, z = c % gx, c // gx % gy, c // (gx * gy)
        rows = [(zz * gy + yy) * gx for zz in range(max(z - 1, 0), min(z + 2, gz))
                for yy in range(max(y - 1, 0), min(y + 2, gy))]
        j = np.concatenate([np.arange(off[r + max(x - 1, 0)], off[r + min(x + 1, gx - 1) + 1]) for r in rows])
        for k0 in range(off[c], off[c + 1], 256):
            k = np.arange(k0, min(k0 + 256, off[c + 1]))
            r2 = 1e-5 + ((p[k][:, None, :] - p[j][None]) ** 2).sum(2)
            r6 = 1.0 / (r2 * r2 * r2)
            e = r6 * r6 - r6
            e[k[:, None] == j[None]] = 0.0
            v[k] = 4.0 * e.sum(1)
    return v


CASES = {
    **{f"{side}_cells_a_side_{n}": (lambda n=n, side=side: uniform(n, n + side), 0.9999 / side)
       for side in (1, 2, 3, 5) for n in (1000, 9001)},
    "droplet_few_cells": (lambda: droplet(9000, 0.0999, 0.5, 1), 0.0999),
    "droplet_filled_grid": (lambda: droplet(60_000, 0.0499, 0.04, 2), 0.0499),   # 8000 cells: chunks of 64
    # cells of 15 to 129 targets side by side, on few cells and on a grid that fills the GPU
    "edges_of_16": (lambda: cells_of([15, 16, 17, 31, 32, 33, 0, 1, 47, 48, 49], 5, 3), 0.19999),
    "edges_of_64": (lambda: cells_of([63, 64, 65, 127, 128, 129, 0, 1, 2, 191, 192, 193, 700] + [6] * 4900, 17, 4),
                    0.9999 / 17),
}


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("name", list(CASES))
def test_law_on_crowded_cells(torch_cuda, ctx, name, order):
    import ljcell

    torch = torch_cuda
    make, width = CASES[name]
    p = make()
    n = len(p)
    x, y, z = (np.ascontiguousarray(p[:, k]) for k in range(3))
    box = ((0, 0, 0), (1, 1, 1))
    g, og = ljcell.grid_from_box(*box, width), O.grid_from_box(*box, width)
    b = ctx.bin(g, dev(torch, x), dev(torch, y), dev(torch, z), order=order)
    v = torch.full((n,), float("nan"), device="cuda")
    ctx.compute_compat(g, b, v)
    ctx.sync()
    ref = law64(og, O.bin_particles(og, x, y, z, order))
    got = np_(v)
    assert np.all(np.isfinite(got))
    rel = np.where(ref == 0, np.abs(got), np.abs((ref - got) / np.where(ref == 0, 1, ref)))
    assert rel.max() <= COMPAT_REL_TOL


@pytest.mark.parametrize("side,n,at", [(5, 2000, 1000), (5, 2000, 1999), (20, 60_000, 12_345), (30, 60_000, 12_345)])
def test_cell_id_outside_the_grid_is_reported(torch_cuda, ctx, side, n, at):
    """Few cells, a filled grid and a sparse one (the two-target kernel)."""
    import ljcell

    torch = torch_cuda
    g = ljcell.grid_from_box((0, 0, 0), (1, 1, 1), 0.9999 / side)
    b = ctx.bin(g, *(dev(torch, np.ascontiguousarray(c)) for c in uniform(n, 5).T))
    for bad in (-1, g.ncells):
        b.cell[at] = bad
        ctx.compute_compat(g, b)
        with pytest.raises(ljcell.LJError) as ei:
            ctx.sync()
        assert ei.value.status == ljcell.LJ_ERANGE
    ctx.sync()
