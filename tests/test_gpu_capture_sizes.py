"""A context warmed up with a larger system captures a smaller one of the same density: the pair stage's scratch,
whose size falls where a warp takes one group of targets more, must not have to grow for it, nor for a sparser
grid, where another walk has more blocks."""
import pytest

pytestmark = pytest.mark.gpu


def binned(torch, ctx, n, per_cell, seed):
    import ljcell

    gen = torch.Generator(device="cuda").manual_seed(seed)
    rc = (per_cell / n) ** (1 / 3)
    g = ljcell.grid_from_box((0, 0, 0), (1, 1, 1), rc)
    return g, ljcell.params(rc), ctx.bin(g, *(torch.rand(n, device="cuda", generator=gen) for _ in range(3)))


def capture(torch, stream, call):
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    graph.replay()
    torch.cuda.synchronize()


@pytest.mark.parametrize("form,large,small", [("plain", (200_000, 10), (149_000, 10)), ("plain", (2_000_000, 10), (1_900_000, 3)),
                                              ("mixed", (200_000, 45), (127_000, 45)), ("mixed", (2_000_000, 45), (1_900_000, 15))])
def test_smaller_pair_stage_under_capture(torch_cuda, form, large, small):
    """(particles, particles per cell) of the warm-up and of the captured system."""
    import ljcell

    torch = torch_cuda
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = ljcell.Context(0, stream)

        def run(g, p, b, rec, out):
            ctx.compute(g, p, b, *out) if form == "plain" else ctx.compute_mixed(g, p, b, rec, *out)

        systems = []
        for n, per_cell in (large, small):
            g, p, b = binned(torch, ctx, n, per_cell, n)
            systems.append((g, p, b, ctx.pack_mixed(g, b), ctx.alloc_outputs(n)))
        run(*systems[0])
        ctx.sync()
    out = ctx.alloc_outputs(small[0])
    g, p, b, rec, _ = systems[1]
    capture(torch, stream, lambda: run(g, p, b, rec, out))
    with torch.cuda.stream(stream):
        run(g, p, b, rec, systems[1][4])
        ctx.sync()
    for got, want in zip(out, systems[1][4]):
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    ctx.close()


def test_ticket_build_under_capture_after_one_launch_builds(torch_cuda):
    """Warmed up with small systems, which one launch builds without any scratch; captured: fewer particles on
    more cells than that launch takes, and the same particles with a set number of scatter passes."""
    import ljcell

    torch = torch_cuda
    stream = torch.cuda.Stream()
    gen = torch.Generator(device="cuda").manual_seed(4)
    xyz = [torch.rand(4096, device="cuda", generator=gen) for _ in range(3)]
    for n, rc, passes in ((3000, 0.0476, 0), (4096, 0.05001, 2)):
        with torch.cuda.stream(stream):
            ctx = ljcell.Context(0, stream)
            ctx.bin(ljcell.grid_from_box((0, 0, 0), (1, 1, 1), 0.0501), *xyz)
            ctx.sync()
        g = ljcell.grid_from_box((0, 0, 0), (1, 1, 1), rc)
        part = [v[:n].contiguous() for v in xyz]
        out, want = ctx.alloc_binned(g, n), ctx.alloc_binned(g, n)
        ctx.set_tuning(0, passes)
        capture(torch, stream, lambda: ctx.bin(g, *part, out=out))
        with torch.cuda.stream(stream):
            ctx.bin(g, *part, out=want)
            ctx.sync()
        for k in ("counts", "offsets", "cell"):
            assert torch.equal(getattr(out, k), getattr(want, k))
        assert torch.equal(out.xyzi.view(torch.int32), want.xyzi.view(torch.int32))
        ctx.close()
