"""Binning in place -- the positions lie in the call's own sorted outputs -- and the bits of x: each of the
three builds (one launch, tickets, segments) gives what it gives for separate inputs, with the sign of every
zero, and the one-launch and segment builds keep the bits of a NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUILDS = {"one_launch": (3000, 0.2), "tickets": (60_000, 0.06), "segments": (4_000_100, 0.0137)}


def points(torch, n, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.rand((n, 3), device="cuda", generator=gen)
    zero = torch.rand(n, device="cuda", generator=gen) < 0.2
    sign = torch.rand(n, device="cuda", generator=gen) < 0.5
    p[:, 0] = torch.where(zero, torch.where(sign, 0.0, -0.0), p[:, 0])
    return p


def same(torch, a, b):
    for k in ("counts", "offsets", "cell", "index"):
        assert torch.equal(getattr(a, k), getattr(b, k)), k
    for k in ("xyzi", "sx", "sy", "sz"):
        assert torch.equal(getattr(a, k).view(torch.int32), getattr(b, k).view(torch.int32)), k


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("name", list(BUILDS))
def test_binning_in_place(torch_cuda, ctx, name, order):
    import ljcell

    torch = torch_cuda
    n, rc = BUILDS[name]
    g = ljcell.grid_from_box((0, 0, 0), (1, 1, 1), rc)
    for seed in range(3):
        p = points(torch, n, 70 + seed)
        cols = [p[:, k].contiguous() for k in range(3)]
        want = ctx.bin(g, *cols, order=order, soa=True)
        i = want.index.long()
        assert torch.equal(want.xyzi[:, :3].contiguous().view(torch.int32), p[i].view(torch.int32))
        soa = ctx.alloc_binned(g, n, order, soa=True)
        for to, c in zip((soa.sx, soa.sy, soa.sz), cols):
            to.copy_(c)
        ctx.bin(g, soa.sx, soa.sy, soa.sz, order=order, out=soa)
        same(torch, soa, want)
        rec = ctx.alloc_binned(g, n, order, soa=True)
        rec.xyzi[:, :3] = p
        flat = rec.xyzi.view(-1)
        ctx.bin(g, flat, flat[1:], flat[2:], stride=4, order=order, out=rec)
        same(torch, rec, want)
    ctx.sync()


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("name", ["one_launch", "segments"])
def test_bits_of_non_finite_x(torch_cuda, ctx, name, order):
    import ljcell

    torch = torch_cuda
    n, rc = BUILDS[name]
    p = points(torch, n, 90)
    odd = np.array([0x7FC00000, 0x7FC12345, 0xFFC00001, 0x7F812345, 0x7F800000, 0xFF800000, 0x00000001, 0x80000001],
                   np.uint32)
    p[100:100 + len(odd), 0] = torch.from_numpy(odd.view(np.float32)).cuda()
    g = ljcell.grid_from_box((0, 0, 0), (1, 1, 1), rc)
    b = ctx.bin(g, *(p[:, k].contiguous() for k in range(3)), order=order)
    with pytest.raises(ljcell.LJError) as ei:
        ctx.sync()
    assert ei.value.status == ljcell.LJ_ERANGE
    i = b.xyzi[:, 3].contiguous().view(torch.int32).long()
    assert torch.equal(torch.sort(i).values, torch.arange(n, device="cuda"))
    assert torch.equal(b.xyzi[:, :3].contiguous().view(torch.int32), p[i].view(torch.int32))
