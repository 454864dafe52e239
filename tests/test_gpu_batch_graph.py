"""The batched step's graph replay after the context's build scratch was replaced: a later, larger build on
the same context frees the buffers whose addresses the graph was captured with, and another context has its
own.  Both have to lead to a new capture: the outputs keep the bits of the plain step, and memory that the
library has given back is left alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def outputs(b):
    e, f, idx, tot = b.alloc_outputs()
    for t in (e, f, idx, tot):
        t.zero_()
    return e, f, idx, tot


def bits(ts):
    return [t.detach().cpu().numpy().view(np.uint8).copy() for t in ts]


def test_graph_replay_after_the_build_scratch_grew(torch_cuda):
    import ljcell

    torch = torch_cuda
    first, second = ljcell.Context(0), ljcell.Context(0)
    b = ljcell.Batch(first, ljcell.batch_workload(nsys=12, seed=21, n_min=50, n_max=4000, nb_min=10, nb_max=60))
    xyz = b.generate()
    plain, out = outputs(b), outputs(b)
    b.run(*xyz, *plain, mode="plain")
    first.sync()
    want = bits(plain)

    def replay():
        for t in out:
            t.zero_()
        b.run(*xyz, *out, mode="graph")
        b.ctx.sync()
        assert all(np.array_equal(w, g) for w, g in zip(want, bits(out)))

    replay()
    # a build that needs more of every buffer: tickets and records, the scan's state, the large-cell list
    n = 2_500_000
    g = ljcell.grid_from_box((0, 0, 0), (1, 1, 1), 0.005)
    x = torch.rand(3 * n, device="cuda")
    first.bin(g, x[:n], x[n:2 * n], x[2 * n:])
    first.sync()
    kept = [torch.full((1 << 20,), 7, dtype=torch.int32, device="cuda") for _ in range(16)]
    replay()
    replay()
    b.ctx = second     # the same plan through another context ...
    replay()
    b.ctx = first
    replay()
    b.ctx = second
    first.close()      # ... which outlives the one it was captured with
    replay()
    assert all(bool((k == 7).all()) for k in kept)
    b.close()
    second.close()
