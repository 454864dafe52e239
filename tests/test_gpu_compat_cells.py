"""The reference law's warp-per-cell kernel at the edges of its tiles: cells of 1 to 33 particles (16
targets a round), stencils of odd ranges and of more candidates than a warp holds at once, grids without
neighbour rows, and the densities on both sides of its dispatch; against the oracle within the
reference's own tolerance."""
import numpy as np
import pytest

import ljoracle as O
from test_gpu_parity import COMPAT_REL_TOL, dev, np_

pytestmark = pytest.mark.gpu

# box, cell width, particles
SHAPES = {
    **{f"one_cell_{n}": (((0, 0, 0), (0.5, 0.5, 0.5)), 0.5, n) for n in (1, 2, 3, 4, 5, 15, 16, 17, 33)},
    "one_row": (((0, 0, 0), (1.0, 0.1, 0.1)), 0.1, 157),
    "list_in_parts": (((0, 0, 0), (0.5, 0.5, 0.5)), 0.1, 9001),      # about 1,900 candidates per cell
    "six_per_cell": (((0, 0, 0), (1.0, 1.0, 1.0)), 0.05, 48_000),
    "below_six_per_cell": (((0, 0, 0), (1.0, 1.0, 1.0)), 0.05, 47_900),
    "few_sparse_cells": (((0, 0, 0), (1.0, 1.0, 1.0)), 0.1, 1500),
}


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("name", list(SHAPES))
def test_compat_cells_edges(torch_cuda, ctx, name, order):
    import ljcell

    torch = torch_cuda
    (lo, hi), width, n = SHAPES[name]
    rng = np.random.default_rng(n)
    p = (np.array(lo, np.float32) + np.array(hi, np.float32) * rng.random((n, 3), dtype=np.float32)).astype(np.float32)
    x, y, z = (np.ascontiguousarray(p[:, k]) for k in range(3))
    g, og = ljcell.grid_from_box(lo, hi, width), O.grid_from_box(lo, hi, width)
    b = ctx.bin(g, dev(torch, x), dev(torch, y), dev(torch, z), order=order)
    v = torch.full((n,), float("nan"), device="cuda")
    ctx.compute_compat(g, b, v)
    ctx.sync()
    ref = O.compat_energy(og, O.bin_particles(og, x, y, z, order))
    got = np_(v)
    assert np.all(np.isfinite(got))
    rel = np.where(ref == 0, np.abs(got), np.abs((ref - got) / np.where(ref == 0, 1, ref)))
    assert rel.max() <= COMPAT_REL_TOL
