"""The cluster walk where a row of cells has several segments (64 cells, from whose start the clusters are
counted): rows of 63 to 129 cells, so that a segment ends inside a row, fills it exactly or is one cell long, and
target ranges that start and end around a segment's first target; the plain form in both within-cell orders and
the mixed form, against the FP64 oracle with the tolerances of test_gpu_parity."""
import numpy as np
import pytest

import ljoracle as O
from test_gpu_parity import ENERGY_SCALED_TOL, FORCE_NORMWISE_TOL, FORCE_SCALED_TOL, dev, np_

pytestmark = pytest.mark.gpu

WIDTH = 0.1
#        cells along x, y, z; particles
SHAPES = {"63": (63, 1, 1, 700), "64": (64, 1, 1, 640), "65": (65, 1, 1, 651), "65_rows": (65, 2, 3, 4001),
          "128_rows": (128, 3, 1, 3900), "129": (129, 1, 1, 1300), "129_rows": (129, 2, 2, 5170),
          "129_thin": (129, 2, 1, 700)}


def system(name, seed):
    import ljcell

    gx, gy, gz, n = SHAPES[name]
    hi = tuple(float(np.float32((c + 0.02) * WIDTH)) for c in (gx, gy, gz))
    rng = np.random.default_rng(seed)
    p = (rng.random((n, 3)) * np.array([gx, gy, gz]) * WIDTH).astype(np.float32)
    g, og = ljcell.grid_from_box((0, 0, 0), hi, WIDTH), O.grid_from_box((0, 0, 0), hi, WIDTH)
    assert tuple(g.dim) == (gx, gy, gz)
    return g, og, [np.ascontiguousarray(p[:, k]) for k in range(3)]


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("name", list(SHAPES))
def test_cluster_walk_over_segments(torch_cuda, ctx, name, order):
    import ljcell

    torch = torch_cuda
    g, og, xyz = system(name, 11 + order)
    n = len(xyz[0])
    p = ljcell.params(WIDTH, sigma=WIDTH / 10)
    ob = O.bin_particles(og, *xyz, order)
    off = ob.offsets
    cuts = sorted({int(np.clip(off[r * g.dim[0] + c] + d, 0, n)) for r in range(g.dim[1] * g.dim[2]) for c in (63, 64, 128)
                   if c < g.dim[0] for d in (-1, 0, 1, 9)} | {0, n})
    ctx.set_tuning(1)
    try:
        b = ctx.bin(g, *(dev(torch, a) for a in xyz), order=order)
        e, f, tot = ctx.compute(g, p, b)
        ctx.sync()
        pairs = 0
        for kb, ke in zip(cuts, cuts[1:]):
            pe, pf, pt = ctx.alloc_outputs(n)
            pe.fill_(float("nan"))
            ctx.compute_range(g, p, b, kb, ke, pe, pf, pt)
            ctx.sync()
            pairs += ljcell.totals_from_tensor(pt)["pairs"]
            assert torch.equal(pe[kb:ke].view(torch.int32), e[kb:ke].view(torch.int32)), (kb, ke)
            assert torch.equal(pf[kb:ke].view(torch.int32), f[kb:ke].view(torch.int32)), (kb, ke)
            assert bool(torch.isnan(pe[:kb]).all()) and bool(torch.isnan(pe[ke:n]).all())
    finally:
        ctx.set_tuning(0)
    ref = O.config_forces(og, ob, WIDTH, 1.0, p.sigma)
    assert ljcell.totals_from_tensor(tot)["pairs"] == ref.pairs == pairs
    fe, ee = ref.force_errors(np_(f)[:n], FORCE_SCALED_TOL), ref.energy_errors(np_(e)[:n], ENERGY_SCALED_TOL)
    assert fe["max_scaled_over_tol"] <= 1.0 and ee["max_scaled_over_tol"] <= 1.0
    assert fe["normwise"] <= FORCE_NORMWISE_TOL


@pytest.mark.parametrize("name", [s for s, (x, y, z, n) in SHAPES.items() if n >= 8 * x * y * z])
def test_mixed_cluster_walk_over_segments(torch_cuda, ctx, name):
    import ljcell

    torch = torch_cuda
    g, og, xyz = system(name, 17)
    n = len(xyz[0])
    p = ljcell.params(WIDTH, sigma=WIDTH / 10)
    b = ctx.bin(g, *(dev(torch, a) for a in xyz))
    e, f, tot = ctx.compute_mixed(g, p, b, ctx.pack_mixed(g, b))
    ctx.sync()
    ob = O.bin_particles(og, *xyz, O.ORDER_X)
    ref = O.mixed_forces(og, ob, *O.pack_mixed(og, ob), WIDTH, 1.0, p.sigma)
    assert ljcell.totals_from_tensor(tot)["pairs"] == ref.pairs
    fe, ee = ref.force_errors(np_(f)[:n]), ref.energy_errors(np_(e)[:n])
    assert fe["max_scaled"] <= FORCE_SCALED_TOL and fe["normwise"] <= FORCE_NORMWISE_TOL
    assert ee["max_scaled"] <= ENERGY_SCALED_TOL
