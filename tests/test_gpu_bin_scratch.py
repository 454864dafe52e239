"""A large build without room for the segment build's own scratch: an allocation that fails, and a capture in
which nothing may be allocated.  Both take the ticket build, with the same results; failures of what that one
needs are reported as before."""
import pytest

pytestmark = pytest.mark.gpu

BOX = ((0, 0, 0), (1, 1, 1))


def points(torch, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.rand(n, device="cuda", generator=gen) for _ in range(3)]


def same(torch, a, b):
    for k in ("counts", "offsets", "cell"):
        assert torch.equal(getattr(a, k), getattr(b, k)), k
    assert torch.equal(a.xyzi.view(torch.int32), b.xyzi.view(torch.int32))


def test_segment_scratch_that_cannot_be_allocated(torch_cuda, ctx):
    import ljcell

    torch = torch_cuda
    xyz, g = points(torch, 4_050_000, 81), ljcell.grid_from_box(*BOX, 0.0135)
    want = ctx.bin(g, *xyz)
    ctx.sync()
    for k in range(1, 6):   # the segment build's scratch, tickets, unsorted records, large-cell list, scan state
        fresh = ljcell.Context(0)
        try:
            ljcell.test_fail_alloc(k)
            if k == 1:
                same(torch, fresh.bin(g, *xyz), want)
            else:
                with pytest.raises(ljcell.LJError) as err:
                    fresh.bin(g, *xyz)
                assert err.value.status == ljcell.LJ_ENOMEM
        finally:
            ljcell.test_fail_alloc(0)
        same(torch, fresh.bin(g, *xyz), want)
        fresh.sync()
        fresh.close()


def test_capture_of_a_grid_with_more_segments(torch_cuda, ctx):
    """A context warmed up with more particles and, apart from those, more cells captures a build of a grid
    with more segments than it has scratch for."""
    import ljcell

    torch = torch_cuda
    stream = torch.cuda.Stream()
    fresh = ljcell.Context(0, stream)
    xyz, g = points(torch, 4_100_000, 82), ljcell.grid_from_box(*BOX, 0.0125)
    want = ctx.bin(g, *xyz)
    ctx.sync()
    fresh.bin(ljcell.grid_from_box(*BOX, 0.0217), *points(torch, 4_200_000, 83))
    fresh.bin(g, *points(torch, 20_000, 84))
    out = fresh.alloc_binned(g, 4_100_000)
    fresh.sync()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        fresh.bin(g, *xyz, out=out)
    for _ in range(2):
        for t in (out.counts, out.offsets, out.cell, out.xyzi):
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        same(torch, out, want)
    fresh.sync()
    del graph
    fresh.close()
