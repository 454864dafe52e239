"""Contexts on several host threads, each binning on a stream of its own: one-launch builds of small systems
and segment builds of large ones, on grids that need more and less shared memory, at the same time.  Every
call succeeds and every result is the one of a single thread."""
import threading

import pytest

pytestmark = pytest.mark.gpu

#        particles, cutoff: cells up to the one-launch build's 8192 and few; segments of 8192 and of 64 cells
SYSTEMS = [(4096, 0.0501), (2000, 0.34), (4_000_000, 0.0025), (4_000_000, 0.0135)]


def test_builds_of_concurrent_threads(torch_cuda):
    import ljcell

    torch = torch_cuda
    jobs = []
    for i, (n, rc) in enumerate(SYSTEMS):
        gen = torch.Generator(device="cuda").manual_seed(60 + i)
        xyz = [torch.rand(n, device="cuda", generator=gen) for _ in range(3)]
        g = ljcell.grid_from_box((0, 0, 0), (1, 1, 1), rc)
        one = ljcell.Context(0)
        b = one.bin(g, *xyz)
        one.sync()
        one.close()
        jobs.append((g, xyz, b))
    torch.cuda.synchronize()
    errors = []
    start = threading.Barrier(2 * len(jobs))

    def work(g, xyz, want, rounds):
        try:
            stream = torch.cuda.Stream()
            ctx = ljcell.Context(0, stream)
            out = ctx.alloc_binned(g, want.n)
            torch.cuda.synchronize()
            start.wait(60)
            for _ in range(rounds):
                ctx.bin(g, *xyz, out=out)
            ctx.sync()
            for k in ("counts", "offsets", "cell"):
                assert torch.equal(getattr(out, k), getattr(want, k)), k
            assert torch.equal(out.xyzi.view(torch.int32), want.xyzi.view(torch.int32))
            ctx.close()
        except BaseException as e:  # noqa: BLE001 - reported by the test's own thread
            errors.append(e)
            start.abort()

    threads = [threading.Thread(target=work, args=(*j, 2000 if j[2].n < 5000 else 40)) for j in jobs for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
    assert not any(t.is_alive() for t in threads)
