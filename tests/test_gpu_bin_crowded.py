"""Crowded cells in the one-launch and the segment builds, against the oracle bit for bit: cells on both sides
of the size from which they are sorted instead of ranked, of the small and the large sort kernel's capacity
and of any block's, several in one segment, equal keys and zeros of both signs; both orders."""
import numpy as np
import pytest

import ljoracle as O
from test_gpu_parity import dev, np_

pytestmark = pytest.mark.gpu

BOX = ((0, 0, 0), (1, 1, 1))


def in_cells(rng, cells, counts, width, levels=0):
    """counts[i] particles in cell cells[i] (x, y, z cell coordinates); levels > 0: that many values of x a cell,
    in a row's first cell among them 0 and -0."""
    c = np.repeat(np.array(cells), counts, axis=0)
    u = 0.02 + 0.96 * rng.random((len(c), 3))
    if levels:
        u[:, 0] = rng.integers(0, levels, len(c)) / (levels + 1.0)
        u[(u[:, 0] == 0) & (c[:, 0] > 0), 0] = 0.02
    p = ((c + u) * width).astype(np.float32)
    zero = p[:, 0] == 0
    p[zero, 0] = np.where(rng.random(int(zero.sum())) < 0.5, np.float32(0.0), np.float32(-0.0))
    return p


def check(torch, ctx, p, width, order):
    import ljcell

    n = len(p)
    x, y, z = (np.ascontiguousarray(p[:, k]) for k in range(3))
    g, og = ljcell.grid_from_box(*BOX, width), O.grid_from_box(*BOX, width)
    ob = O.bin_particles(og, x, y, z, order)
    b = ctx.bin(g, *(dev(torch, a) for a in (x, y, z)), order=order, soa=True, cells=True)
    ctx.sync()
    np.testing.assert_array_equal(np_(b.counts), ob.counts)
    np.testing.assert_array_equal(np_(b.offsets), ob.offsets)
    r = np_(b.xyzi)[:n]
    np.testing.assert_array_equal(r[:, 3].view(np.int32), ob.perm)
    np.testing.assert_array_equal(r[:, :3].view(np.int32), p[ob.perm].view(np.int32))
    np.testing.assert_array_equal(np_(b.cell)[:n], ob.cell_sorted)
    np.testing.assert_array_equal(np_(b.index)[:n], ob.perm)
    np.testing.assert_array_equal(np.stack([np_(t)[:n] for t in (b.sx, b.sy, b.sz)], 1).view(np.int32),
                                  r[:, :3].view(np.int32))
    np.testing.assert_array_equal(np_(b.cells), np.stack([ob.counts, ob.offsets[:-1]], 1))


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("levels", [0, 7])
@pytest.mark.parametrize("counts", [[511], [512], [513], [1024], [1025], [4096], [513, 1, 600, 512, 2047],
                                    [513] * 7, [0, 1500, 0, 2000, 3]])
def test_one_launch_build(torch_cuda, ctx, counts, levels, order):
    rng = np.random.default_rng(len(counts) + sum(counts) + order)
    p = in_cells(rng, [(i % 3, i // 3, i % 2) for i in range(len(counts))], counts, 0.3333, levels)
    check(torch_cuda, ctx, p[rng.permutation(len(p))], 0.3333, order)


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("levels", [0, 9])
@pytest.mark.parametrize("name", ["as_large_as_a_block", "too_large_for_a_block"])
def test_segment_build(torch_cuda, ctx, name, levels, order):
    """4 million uniform particles in the lower half of 74^3 cells (segments of 128 cells) and crowded cells in
    the upper half, each in a segment of its own, and three that share one."""
    rng = np.random.default_rng(7 + order)
    width = 0.0135
    p = rng.random((4_000_000, 3), dtype=np.float32) * np.array([1, 1, 0.5], np.float32)
    counts = [511, 512, 513, 1024, 2047, 2048, 2049, 5000, 10239, 10240 if name == "as_large_as_a_block" else 10241]
    cells = [(0 if i % 2 else 40, 5 * i, 50) for i in range(len(counts))]
    cells += [(3, 7, 60), (4, 7, 60), (9, 7, 60)]
    q = in_cells(rng, cells, counts + [600, 700, 1400], width, levels)
    p = np.concatenate([p, q])
    check(torch_cuda, ctx, p[rng.permutation(len(p))], width, order)


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("levels", [0, 5])
def test_segments_too_large_for_a_block(torch_cuda, ctx, levels, order):
    """Segments of 13,000 to 60,000 records whose cells are ranked (a block of 20^3 cells at 400 each, reaching to
    x = 0), others whose cells are sorted, and one that holds both, among 800,000 uniform particles."""
    rng = np.random.default_rng(17 + order)
    width = 0.0125
    cells = [(i, j, k) for k in range(30, 50) for j in range(30, 50) for i in range(20)]
    counts = list(rng.integers(380, 420, len(cells)))
    cells += [(40, 10, 5), (41, 10, 5), (42, 10, 5), (60, 70, 70), (3, 2, 1), (4, 2, 1), (5, 2, 1)]
    counts += [15_000, 600, 40, 25_000, 511, 9000, 2000]
    p = np.concatenate([in_cells(rng, cells, counts, width, levels), rng.random((800_000, 3), dtype=np.float32)])
    assert len(p) >= 4_000_000
    check(torch_cuda, ctx, p[rng.permutation(len(p))], width, order)
