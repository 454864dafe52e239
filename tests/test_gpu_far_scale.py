"""The candidates that fill up a list lie beyond every particle: a system scaled by a power of two, its box as
large as 2^61 or as small as 2^-50, has the same pairs, energies bit for bit and forces scaled exactly, and a
particle that sits at a round far coordinate is nobody's partner twice."""
import numpy as np
import pytest

from test_gpu_parity import np_

pytestmark = pytest.mark.gpu


def system(torch, n, seed, scale):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.rand(n, device="cuda", generator=gen) * scale for _ in range(3)]


@pytest.mark.parametrize("power", [60, 61, -50])
@pytest.mark.parametrize("order", [0, 1])
def test_cluster_walk_in_a_scaled_box(torch_cuda, ctx, power, order):
    import ljcell

    n, rc = 9001, 0.1111
    got = []
    for s in (1.0, 2.0 ** power):
        g = ljcell.grid_from_box((0, 0, 0), (s, s, s), float(np.float32(rc)) * s)
        p = ljcell.params(g.width, sigma=float(np.float32(0.05)) * s)
        b = ctx.bin(g, *system(torch_cuda, n, 3, s), order=order)
        ctx.set_tuning(1)
        try:
            e, f, t = ctx.compute(g, p, b)
            ctx.sync()
        finally:
            ctx.set_tuning(0)
        got.append((np_(e), np_(f).astype(np.float64) * s, ljcell.totals_from_tensor(t)))
    assert got[0][2]["pairs"] == got[1][2]["pairs"]
    assert np.array_equal(got[0][0].view(np.int32), got[1][0].view(np.int32))
    assert np.array_equal(got[0][1], got[1][1])


def test_law_with_a_particle_far_away(torch_cuda, ctx):
    """Few cells of a box that reaches 1.5e18, one particle at (1e18, 1e18, 1e18): every distance is so large
    that every energy is an exact 0."""
    import ljcell

    torch = torch_cuda
    n = 3001
    xyz = system(torch, n, 5, 1.5e18)
    for v in xyz:
        v[7] = 1e18
    g = ljcell.grid_from_box((0, 0, 0), (1.5e18,) * 3, 3e17)
    v = ctx.compute_compat(g, ctx.bin(g, *xyz))
    ctx.sync()
    assert bool((v == 0).all())
