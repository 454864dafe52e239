"""The pair kernel that the default takes on grids whose rows of cells hold few particles, told by the bits of its
results: the cluster walk only where rows fill its clusters, and on small systems."""
import pytest

pytestmark = pytest.mark.gpu

#        cells along x, y and z, particles per cell, order -> kernel of the default
CASES = [(1, 80, 6.2, 1, 10), (1, 80, 7.9, 1, 10), (1, 80, 8.1, 1, 1), (2, 60, 6.2, 1, 1), (1, 60, 6.2, 1, 1),
         (1, 60, 17.5, 0, 11), (1, 60, 18.5, 0, 1), (2, 60, 8.5, 0, 11), (2, 60, 9.5, 0, 1), (3, 60, 6.2, 0, 1),
         (1, 60, 6.2, 0, 1), (20, 20, 5.9, 1, 10), (20, 20, 6.2, 1, 1), (20, 20, 5.9, 0, 11), (20, 20, 1.9, 1, 12)]


@pytest.mark.parametrize("gx,m,per_cell,order,kernel", CASES)
def test_default_kernel_by_rows(torch_cuda, ctx, gx, m, per_cell, order, kernel):
    import ljcell

    torch = torch_cuda
    w = 0.1
    hi = tuple((c + 0.01) * w for c in (gx, m, m))
    g = ljcell.grid_from_box((0, 0, 0), hi, w)
    assert tuple(g.dim) == (gx, m, m)
    gen = torch.Generator(device="cuda").manual_seed(int(10 * per_cell) + gx)
    n = int(per_cell * g.ncells)
    xyz = [torch.rand(n, device="cuda", generator=gen) * h for h in hi]
    p = ljcell.params(w)
    b = ctx.bin(g, *xyz, order=order)
    got = {}
    try:
        for k in (0, 1, 10, 11, 12):
            ctx.set_tuning(k)
            e, f, _ = ctx.compute(g, p, b)
            ctx.sync()
            got[k] = torch.cat([e[:n], f[:n].reshape(-1)]).view(torch.int32)
    finally:
        ctx.set_tuning(0)
    assert torch.equal(got[0], got[kernel])
    others = {1, 10, 11, 12} - {kernel} if order else {1, 11} - {kernel}
    assert not any(torch.equal(got[0], got[k]) for k in others)


def test_slab_rule_is_the_default_rule():
    """The slab's rule, which sees its own layers, agrees with the cases above (no GPU work)."""
    from ljcell.slab import SlabDomain, pair_kernel_for

    class Grid:
        width, origin = 0.1, (0.0, 0.0, 0.0)

    for gx, m, per_cell, order, kernel in CASES:
        Grid.dim = (gx, m, m)
        k = pair_kernel_for(SlabDomain.of(Grid, 0, 1), int(per_cell * gx * m * m), order)
        assert k == kernel or (order == 0 and k != 1 and kernel == 11)
