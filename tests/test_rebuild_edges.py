"""The list rebuild at the edges of its search: every pair list is compared
with the FP64 oracle's (bit-exact order), for scenes that reach the grid's
border cells, the cut rows and end cells of each level, hits beyond the
search's lists, the last cell that also holds out-of-box subspheres, and
scenes of a few subspheres."""
import numpy as np
import pytest

import nbc
import oracle
import scenegen as sg

pytestmark = pytest.mark.gpu


def _spheres(pos, rad, lo, hi, thresh=1e-6, bl=2400, **kw):
    K = len(pos)
    m = 2650 * 4 / 3 * np.pi * rad ** 3
    inertia = 0.4 * m * rad * rad
    params = sg.default_params(StepSize=1e-9, EndStep=1, Thresh=thresh, Gravity=0.0, Ymod=1e3, BranchLmtLen=bl)
    sg.set_world_box(params, lo, hi)
    return sg.assemble(params, pos, np.tile([0, 0, 0, 1.0], (K, 1)), np.zeros((K, 3)), np.zeros((K, 3)),
                       np.stack([inertia, inertia, inertia, m], 1), [np.zeros((1, 3))] * K,
                       [np.array([x]) for x in rad], [np.array([x]) for x in m], **kw)


def _box(n, seed, levels, spread=1.0, cell_scale=1.0, dense=1.0):
    """n spheres of radii 0.3 .. 2.4 mm anywhere in a box (some outside it for
    spread > 1), on `levels` grid levels with cells of cell_scale times three
    radii."""
    rng = np.random.default_rng(seed)
    rad = np.exp(rng.uniform(np.log(0.3e-3), np.log(2.4e-3), n))
    side = max(4e-3, dense * 1.6e-3 * n ** (1 / 3))
    lo, hi = np.array([-0.2, 0.1, 3.0]), np.array([-0.2, 0.1, 3.0]) + side * np.array([1.0, 0.7, 1.3])
    mid = 0.5 * (lo + hi)
    pos = mid + (rng.random((n, 3)) - 0.5) * (hi - lo) * spread
    sc = _spheres(pos, rad, lo, hi)
    if levels > 1:
        edges = np.quantile(rad, np.linspace(1, 0, levels + 1)[1:-1])
        lv = (rad[:, None] <= edges[None, :]).sum(1).astype(np.int32)
        cell = np.array([3 * cell_scale * rad[lv == l].max() if (lv == l).any() else 1e-3 for l in range(levels)])
        sc["levels"] = {"level": lv, "cell": cell}
    return sc


def _same_list(sc, precision):
    e = nbc.Engine([sc], precision=precision, use_graph=False)
    e.step(1)
    e.sync()
    o = oracle.OracleScene(sc, threads=4)
    o.step(1)
    assert np.array_equal(e.subspheres()["part_fix"], o.sub()["part_fix"]), "sort order"
    (la, lb), (oa, ob) = e.pairs(), o.pairs()
    assert np.array_equal(la, oa) and np.array_equal(lb, ob), "pair list"
    bl = sc["params"]["BranchLmtLen"]
    for x, y in zip(e.rows(bl=bl), o.rows()):
        assert np.array_equal(x, y), "rows"
    e.close()
    return len(la)


@pytest.mark.parametrize("n,levels,kw", [
    (1, 1, {}), (2, 1, {"dense": 0.3}), (7, 2, {"dense": 0.3}), (33, 3, {}), (129, 1, {"spread": 1.3}),
    (700, 1, {}), (1500, 6, {}), (1500, 4, {"cell_scale": 1.7}), (1500, 3, {"cell_scale": 0.6}),
    (2000, 5, {"spread": 1.2}), (900, 4, {"dense": 0.35}), (400, 1, {"dense": 0.25})])
def test_lists_equal_the_oracle(n, levels, kw):
    pairs = _same_list(_box(n, 100 + n + levels, levels, **kw), "f64")
    if n > 100:
        assert pairs > n


def test_out_of_box_neighbours_of_the_last_cell():
    """Subspheres that have just left the box through its upper corner: those
    inside list them in their front rows, no back entry exists, and the
    contact acts on the listing subsphere only (src/dem_grid.cu:466-552: an
    out-of-box subsphere does not search)."""
    r = 1e-3
    lo, hi = np.zeros(3), np.full(3, 9e-3)     # three cells of 3 r and the padding
    near = hi - np.array([[0.3, 0.4, 0.2], [0.9, 2.1, 0.5], [2.5, 2.5, 2.5], [0.2, 0.2, 1.9]]) * r
    out = hi + np.array([[0.4, 0.3, 0.5], [0.1, 0.2, 0.3], [9.0, 9.0, 9.0]]) * r
    rng = np.random.default_rng(5)
    bulk = rng.uniform(0.5e-3, 5e-3, (40, 3))
    pos = np.concatenate([bulk, near, out])
    sc = _spheres(pos, np.full(len(pos), r), lo, hi)
    n = _same_list(sc, "f64")
    e = nbc.Engine([sc], precision="f64")
    e.step(1)
    a, b = e.pairs()
    fix = e.subspheres()["part_fix"]
    lost = fix[b] >= len(bulk) + len(near)
    assert lost.sum() >= 3 and n > 40
    e.step(3)
    e.sync()
    o = oracle.OracleScene(sc)
    o.step(4)
    f, _ = e.sub_forces()
    of = o.sub_forces()
    ref = of["fc"] + of["fw"]
    assert np.abs(f - ref).max() <= 1e-10 * np.abs(ref).max()
