"""The passes of nbc_cell_sort_noalloc where they can go wrong: digits of 1 to
9 bits in one to four passes, sizes around a tile of 2,048 keys and up to the
largest, every key in one cell, and a call inside a captured graph.  Against a
numpy hash and stable sort; integer outputs: bit-exact."""
import numpy as np
import pytest

import nbc
from test_zz_no_alloc import numpy_cell_sort

pytestmark = pytest.mark.gpu


def case(dims, n, one_cell=False):
    rng = np.random.default_rng(n)
    g = nbc.GridDesc()
    g.cell = 2.0 ** -10
    for a in range(3):
        g.origin[a] = -g.cell
        g.dims[a] = dims[a]
        g.box_lo[a] = 0.0
        g.box_hi[a] = max(dims[a] - 2, 1) * g.cell
    span = np.array([g.box_hi[a] for a in range(3)])
    pos = np.full((n, 3), 0.25 * g.cell) if one_cell else rng.uniform(-0.02, 1.02, (n, 3)) * span
    return g, pos


def sort(g, dpos, n, stream=0):
    import torch

    perm = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    key = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    nbc.cell_sort_noalloc(dpos.data_ptr(), n, g, perm.data_ptr(), key.data_ptr(), stream)
    return perm, key


@pytest.mark.parametrize("dims", [(1, 1, 1), (8, 8, 8), (8, 8, 9), (64, 64, 64), (64, 64, 65), (512, 512, 512),
                                  (512, 512, 513), (1024, 1024, 1024)])   # 1, 9, 10, 18, 19, 27, 28 and 30 bits
@pytest.mark.parametrize("n", [1, 33, 2047, 2048, 2049, 6145])
def test_digits_and_tile_edges(dims, n):
    import torch

    g, pos = case(dims, n)
    perm, key = sort(g, torch.from_numpy(pos).cuda(), n)
    wp, wk = numpy_cell_sort(pos, g)
    assert np.array_equal(perm.cpu().numpy(), wp) and np.array_equal(key.cpu().numpy(), wk)


@pytest.mark.parametrize("dims,one_cell", [((50, 50, 50), False), ((50, 50, 50), True), ((200, 200, 200), False)])
def test_largest_size_twice(dims, one_cell):
    import torch

    n = nbc.NOALLOC_MAX_N
    g, pos = case(dims, n, one_cell)
    dpos = torch.from_numpy(pos).cuda()
    wp, wk = numpy_cell_sort(pos, g)
    for _ in range(2):
        perm, key = sort(g, dpos, n)
        assert np.array_equal(perm.cpu().numpy(), wp) and np.array_equal(key.cpu().numpy(), wk)


def test_captured_call_replays():
    import torch

    g, pos = case((40, 40, 40), 5003)
    dpos = torch.from_numpy(pos).cuda()
    sort(g, dpos, 5003)   # the first call on a device is not captured
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        perm, key = sort(g, dpos, 5003, torch.cuda.current_stream().cuda_stream)
    pos2 = pos[::-1].copy()
    for p in (pos, pos2):   # new positions in the same buffer: the replay sorts those
        dpos.copy_(torch.from_numpy(p))
        graph.replay()
        torch.cuda.synchronize()
        wp, wk = numpy_cell_sort(p, g)
        assert np.array_equal(perm.cpu().numpy(), wp) and np.array_equal(key.cpu().numpy(), wk)
