"""The binning by segments of cells (large systems) against the oracle, bit for bit: the smallest size
that takes it, ragged sizes and grids (a last segment of a few cells), both orders, point3d input with
every optional output, segments for the large sort kernel, particles crowded into few segments (the
ticket kernels behind the gate), nearly sorted input and points outside the box; and the binning of small systems by one block."""
import numpy as np
import pytest

import ljoracle as O
from test_gpu_parity import dev, np_

pytestmark = pytest.mark.gpu

UNIT = ((0, 0, 0), (1, 1, 1))


def uniform(n, seed):
    rng = np.random.default_rng(seed)
    return rng.random((n, 3), dtype=np.float32)


def positions(name):
    if name == "smallest":
        return uniform(4_000_000, 1), UNIT, 0.0135
    if name == "ragged":          # 82 x 118 x 6 cells, a partial last segment
        p = uniform(4_000_001, 2) * np.array([0.82, 1.18, 0.06], np.float32)
        return p.astype(np.float32), ((0, 0, 0), (0.82, 1.18, 0.06)), 0.01
    if name == "sparse":          # 64 million cells, segments of 8192 cells
        return uniform(4_050_000, 3), UNIT, 0.0025
    if name == "slab":            # half the particles in 1/16 of the box: segments beyond the small sort kernel
        p = uniform(4_100_000, 4)
        p[::2, 2] *= np.float32(1 / 16)
        return p, UNIT, 0.0125
    if name == "crowded":         # 1,200,000 particles in one corner of 8^3 cells: the gate opens
        p = uniform(4_200_000, 5)
        p[:1_200_000] *= np.float32(0.1)
        return p, UNIT, 0.0125
    if name == "one_cell":        # 20,000 particles in a single cell
        p = uniform(4_020_000, 6)
        p[:20_000] = np.float32(0.41) + p[:20_000] * np.float32(0.003)
        return p, UNIT, 0.0125
    if name == "sorted":          # the order of a previous binning
        p = uniform(4_000_500, 7)
        c = np.minimum((p / np.float32(0.0125)).astype(np.int32), 79)
        return p[np.lexsort((p[:, 0], (c[:, 2] * 80 + c[:, 1]) * 80 + c[:, 0]))], UNIT, 0.0125
    if name == "outside":
        p = uniform(4_050_000, 8) * np.float32(1.5) - np.float32(0.25)
        return p.astype(np.float32), UNIT, 0.0125
    raise KeyError(name)


@pytest.mark.parametrize("name,order", [("smallest", 1), ("ragged", 0), ("ragged", 1), ("sparse", 1), ("slab", 0), ("slab", 1),
                                        ("crowded", 0), ("crowded", 1), ("one_cell", 1), ("sorted", 1),
                                        ("outside", 0), ("outside", 1)])
def test_segment_binning_bit_exact(torch_cuda, ctx, name, order):
    import ljcell

    torch = torch_cuda
    p, (lo, hi), rc = positions(name)
    n = len(p)
    x, y, z = (np.ascontiguousarray(p[:, k]) for k in range(3))
    g, og = ljcell.grid_from_box(lo, hi, rc), O.grid_from_box(lo, hi, rc)
    ob = O.bin_particles(og, x, y, z, order)
    aos = dev(torch, p.reshape(-1))
    for stride in (1, 3):
        out = ctx.alloc_binned(g, n, order, soa=stride == 3, cells=stride == 3)
        for t in (out.counts, out.offsets, out.cell):
            t.fill_(-7)
        d = (aos, aos[1:], aos[2:]) if stride == 3 else tuple(dev(torch, a) for a in (x, y, z))
        ctx.bin(g, *d, stride=stride, order=order, out=out)
        ctx.sync()
        np.testing.assert_array_equal(np_(out.counts), ob.counts)
        np.testing.assert_array_equal(np_(out.offsets), ob.offsets)
        r = np_(out.xyzi)
        np.testing.assert_array_equal(r[:, 3].view(np.int32), ob.perm)
        np.testing.assert_array_equal(r[:, :3], np.stack([ob.sx, ob.sy, ob.sz], 1))
        np.testing.assert_array_equal(np_(out.cell), ob.cell_sorted)
        if stride == 3:
            np.testing.assert_array_equal(np_(out.index), ob.perm)
            np.testing.assert_array_equal(np.stack([np_(out.sx), np_(out.sy), np_(out.sz)], 1), r[:, :3])
            np.testing.assert_array_equal(np_(out.cells), np.stack([ob.counts, ob.offsets[:-1]], 1))


def test_segment_binning_reports_a_non_finite_position(torch_cuda, ctx):
    import ljcell

    torch = torch_cuda
    p = uniform(4_010_000, 9)
    p[123_456, 1] = np.inf
    g = ljcell.grid_from_box(*UNIT, 0.02)
    ctx.bin(g, *(dev(torch, p[:, k].copy()) for k in range(3)))
    with pytest.raises(ljcell.LJError) as ei:
        ctx.sync()
    assert ei.value.status == ljcell.LJ_ERANGE
    ctx.sync()


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("n,box,rc", [(1, 1.0, 0.25), (31, 1.0, 0.25), (1000, 1.0, 0.25), (1025, 1.0, 0.3), (4095, 1.0, 0.05),
                                      (4096, 1.0, 0.0501), (4097, 1.0, 0.05), (3000, 1.0, 0.0496), (777, 1.0, 1.0),
                                      (4096, 0.1, 0.05), (2000, 3.0, 0.151)])
def test_small_system_binning_bit_exact(torch_cuda, ctx, n, box, rc, order):
    """One block bins systems of up to 4096 particles and 8192 cells: both sides of its limits, cell
    counts that are no multiple of four, all particles in one cell, particles beyond the box, and equal x
    (-0 among them)."""
    import ljcell

    torch = torch_cuda
    p = uniform(n, n + order) * np.float32(box)
    p[::7, 0] = np.float32(0.0)
    p[::14, 0] = np.float32(-0.0)
    p[::5, 1] -= np.float32(0.1)
    x, y, z = (np.ascontiguousarray(p[:, k]) for k in range(3))
    g, og = ljcell.grid_from_box(*UNIT, rc), O.grid_from_box(*UNIT, rc)
    ob = O.bin_particles(og, x, y, z, order)
    aos = dev(torch, p.reshape(-1))
    for stride in (1, 3):
        d = (aos, aos[1:], aos[2:]) if stride == 3 else tuple(dev(torch, a) for a in (x, y, z))
        b = ctx.bin(g, *d, stride=stride, order=order, soa=stride == 3, cells=stride == 3)
        ctx.sync()
        np.testing.assert_array_equal(np_(b.counts), ob.counts)
        np.testing.assert_array_equal(np_(b.offsets), ob.offsets)
        r = np_(b.xyzi)[:n]
        np.testing.assert_array_equal(r[:, 3].view(np.int32), ob.perm)
        np.testing.assert_array_equal(r[:, :3].view(np.int32), p[ob.perm].view(np.int32))
        np.testing.assert_array_equal(np_(b.cell)[:n], ob.cell_sorted)
        if stride == 3:
            np.testing.assert_array_equal(np_(b.cells), np.stack([ob.counts, ob.offsets[:-1]], 1))
            np.testing.assert_array_equal(np_(b.index)[:n], ob.perm)
