"""Pair lists of subspheres whose coordinates lie on the faces of grid cells, or
one representable number beside them.  The sort's cell is the floor of a
quotient, and (x - origin) / cell and (x - origin) * (1 / cell) round to
different sides of an integer there; lattices at rest with round radii are full
of such coordinates.  Compared with the FP64 oracle: lists bit for bit, forces
to rounding."""
import numpy as np
import pytest

import nbc
import oracle
from test_rebuild_edges import _box, _spheres

pytestmark = pytest.mark.gpu


def _grid(sc):
    """Origin and cell size of the single-level grid."""
    p = sc["params"]
    cell = 3.0 * sc["sub"]["radius"].max()
    return np.array([p["WorldOrigin_" + a] for a in "xyz"]) - cell, cell


def _rounded_apart(sc):
    """Subspheres that the product puts into another cell than the quotient."""
    org, cell = _grid(sc)
    x = sc["sub"]["pos"] - org
    return (np.floor(x / cell) != np.floor(x * (1.0 / cell))).any(1)


def _lattice(r, spacing, dims, nudge=0, fill=1.0, levels=1):
    """A cubic lattice from the origin on, its coordinates moved by `nudge`
    representable numbers; fill < 1: spheres of radius fill * r, and one of
    radius r beside them that sets the cell."""
    g = np.stack(np.meshgrid(*[np.arange(d) for d in dims], indexing="ij"), -1).reshape(-1, 3)
    pos = spacing * r * g
    for _ in range(abs(nudge)):
        pos = np.nextafter(pos, np.inf if nudge > 0 else -np.inf)
    rad = np.full(len(pos), r)
    if fill < 1.0:
        rad[:] = fill * r
        pos = np.concatenate([pos, [pos.max(0) + 4 * r]])
        rad = np.append(rad, r)
    sc = _spheres(pos, rad, np.minimum(pos.min(0), 0.0), pos.max(0) + 3 * r, thresh=1e-3 * r)
    if levels > 1:
        lv = (np.arange(len(pos)) % levels).astype(np.int32)
        cell = 3 * rad.max() * (1.0 - 0.25 * np.arange(levels))
        sc["sub"]["radius"] = sc["sub"]["radius"] * (1.0 - 0.25 * lv)
        sc["levels"] = {"level": lv, "cell": cell}
    return sc


def _check(e, s, sc):
    o = oracle.OracleScene(sc, threads=4)
    o.step(1)
    assert np.array_equal(e.subspheres(s)["part_fix"], o.sub()["part_fix"]), "sort order"
    (la, lb), (oa, ob) = e.pairs(s), o.pairs()
    assert (la != lb).all(), "a subsphere lists itself"
    assert len({(a, b) if a < b else (b, a) for a, b in zip(la.tolist(), lb.tolist())}) == len(la), "a pair twice"
    assert np.array_equal(la, oa) and np.array_equal(lb, ob), "pair list"
    bl = sc["params"]["BranchLmtLen"]
    (row, ng, ni), (orow, ong, oni) = e.rows(s, bl=bl), o.rows()
    assert np.array_equal(ng, ong), "front rows"
    pairs = set(zip(oa.tolist(), ob.tolist()))
    for i in range(len(ng)):
        assert np.array_equal(row[i, :ng[i]], orow[i, :ng[i]]), "front row"
        # (of two subspheres a cell apart the partner alone may list the other:
        # an entry that refers to no pair, which the engine leaves out)
        back = [j for j in orow[i, bl - oni[i]:][::-1].tolist() if (j, i) in pairs]
        assert row[i, bl - ni[i]:][::-1].tolist() == back, "back row"
    return o


def _list(sc):
    e = nbc.Engine([sc], precision="f64", use_graph=False)
    e.step(1)
    e.sync()
    o = _check(e, 0, sc)
    e.close()
    return o


@pytest.mark.parametrize("dims", [(3, 3, 110), (3, 110, 3), (110, 3, 3)])
@pytest.mark.parametrize("r", [1e-3, 1.5e-3, 5e-3, 0.05])
@pytest.mark.parametrize("nudge", [-1, 0, 1])
@pytest.mark.parametrize("spacing", [2.0, 3.0])   # neighbours in reach, and at its very end
def test_lattice_lists(r, dims, nudge, spacing):
    sc = _lattice(r, spacing, dims, nudge)
    assert nudge or spacing != 2.0 or _rounded_apart(sc).any()
    _list(sc)


@pytest.mark.parametrize("r", [2.5e-3, 0.05])
@pytest.mark.parametrize("levels", [1, 2])
def test_long_rows(r, levels):
    """More than the 64 back entries that the search keeps per subsphere."""
    sc = _lattice(r, 0.75, (6, 4, 90), levels=levels)
    assert levels > 1 or _rounded_apart(sc).any()
    assert _list(sc).rows()[2].max() > 64


@pytest.mark.parametrize("r", [1.5e-3, 0.05])
def test_lattice_leaves_the_box(r):
    """Its upper end outside: the last cell's members are listed by those whose
    stencil holds that cell, and list nobody."""
    sc = _lattice(r, 2.0, (4, 4, 60))
    p, hi = sc["params"], sc["sub"]["pos"].max(0)
    for a, h in zip("xyz", hi - 2 * r):
        p["WorldSize_" + a] = p["BoxUpLmt_" + a] = h
    assert _rounded_apart(sc).any()
    _list(sc)


@pytest.mark.parametrize("n,levels", [(300, 1), (900, 3)])
def test_box_beyond_the_grid(n, levels):
    """A box larger than the grid: subspheres outside the grid are in its border
    cells, their stencils are not."""
    sc = _box(n, 77 + n, levels, spread=1.6)
    p = sc["params"]
    for a in "xyz":
        p["BoxLowLmt_" + a] -= 1.0
        p["BoxUpLmt_" + a] += 1.0
    _list(sc)


@pytest.mark.parametrize("dims", [(3, 3, 70), (3, 70, 3)])
@pytest.mark.parametrize("r", [1.5e-3, 0.05])
@pytest.mark.parametrize("levels", [2, 3])
def test_lattice_lists_on_levels(r, dims, levels):
    _list(_lattice(r, 2.0, dims, levels=levels))


def test_lattices_in_a_batch():
    scenes = [_lattice(1.5e-3, 2.0, (3, 3, 60)), _box(300, 9, 1), _lattice(0.01, 2.0, (3, 60, 3)),
              _lattice(0.05, 2.0, (3, 3, 40), levels=2)]
    e = nbc.Engine(scenes, precision="mixed", use_graph=False)
    e.step(1)
    e.sync()
    for s, sc in enumerate(scenes):
        _check(e, s, sc)
    e.close()


@pytest.mark.parametrize("dims", [(3, 3, 110), (3, 110, 3)])
def test_touching_lattice_forces(dims):
    """Neighbours overlap by 2e-4 of the spacing; a pair listed twice would
    push twice."""
    sc = _lattice(1.5e-3, 1.0, dims, fill=0.5001)
    assert _rounded_apart(sc).any()
    e = nbc.Engine([sc], precision="f64")
    e.step(1)
    e.sync()
    o = _check(e, 0, sc)
    f, _ = e.sub_forces()
    of = o.sub_forces()
    ref = of["fc"] + of["fw"]
    assert np.abs(ref).max() > 0
    assert np.abs(f - ref).max() <= 1e-10 * np.abs(ref).max()
    a, b, c = dims
    assert e.contact_counts()[1] == (a - 1) * b * c + a * (b - 1) * c + a * b * (c - 1)
    e.close()


def test_rebuilds_on_faces_inside_the_step_loop():
    """Two lattices that approach along x, their y and z on faces: a rebuild at
    every step, with lists that outgrow their region on the way."""
    r = 1.5e-3
    sc = _lattice(r, 2.0, (6, 3, 60))
    x = sc["sub"]["pos"][:, 0]
    right = x > 5 * r
    for p in (sc["sub"]["pos"], sc["clump"]["pos"]):
        p[right, 0] += 2.1 * r
    sc["clump"]["vel"][right, 0] = -0.02 * r / sc["params"]["StepSize"]
    for k in ("WorldSize_x", "BoxUpLmt_x"):
        sc["params"][k] += 4 * r
    assert _rounded_apart(sc).any()
    a = nbc.Engine([sc], precision="f64", pair_slack=1.0)
    b = nbc.Engine([sc], precision="f64", pair_slack=4.0, use_graph=False)
    a.step(1)
    first = a.info()["device_bytes"]
    for n in (20, 40, 35):
        a.step(n)
    a.sync()
    b.step(96)
    b.sync()
    assert a.info()["device_bytes"] > first, "the lists did not outgrow their region"
    o = oracle.OracleScene(sc, threads=4)
    o.step(96)
    for e in (a, b):
        (la, lb), (oa, ob) = e.pairs(), o.pairs()
        assert np.array_equal(la, oa) and np.array_equal(lb, ob)
        assert e.stats()["rebuilds"] == o.rebuilds
    for k in ("pos", "vel", "quat", "angvel"):
        assert np.array_equal(a.clumps()[k], b.clumps()[k])


def test_batch_rebuilds_some_scenes_on_faces():
    """Lattices that move along x at different speeds, so that most rebuilds are
    of some of the scenes: each as it is alone, and as the oracle has it."""
    scenes = []
    for k, (r, spacing, dims) in enumerate([(1.5e-3, 2.0, (5, 3, 60)), (2.5e-3, 3.0, (4, 4, 60)), (0.05, 2.0, (4, 60, 3)),
                                            (1.5e-3, 1.0, (4, 3, 40))]):
        sc = _lattice(r, spacing, dims, fill=0.5001 if spacing == 1.0 else 1.0, levels=2 if k == 2 else 1)
        sc["params"]["StepSize"] = 1e-9
        sc["clump"]["vel"][:, 0] = (k + 1) * 0.17e-3 * r / sc["params"]["StepSize"] * np.linspace(1.0, 0.2, len(sc["clump"]["vel"]))
        scenes.append(sc)
    both = nbc.Engine(scenes, precision="f64", pair_slack=3.0)
    both.step(50)
    both.sync()
    counts = set()
    for s, sc in enumerate(scenes):
        e = nbc.Engine([sc], precision="f64", pair_slack=3.0)
        e.step(50)
        e.sync()
        o = oracle.OracleScene(sc, threads=4)
        o.step(50)
        for k in ("pos", "vel", "quat", "angvel", "force", "torque"):
            assert np.array_equal(both.clumps(s)[k], e.clumps()[k]), (s, k)
        assert both.stats(s) == e.stats() and e.stats()["rebuilds"] == o.rebuilds
        counts.add(o.rebuilds)
        for x, y in zip(both.rows(s, bl=2400), e.rows(bl=2400)):
            assert np.array_equal(x, y)
        (la, lb), (oa, ob) = both.pairs(s), o.pairs()
        assert np.array_equal(la, oa) and np.array_equal(lb, ob)
    assert len(counts) > 2


@pytest.mark.parametrize("levels", [1, 2, 4])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("side", [-1, 1])
def test_around_the_end_of_the_grid(levels, axis, side):
    """A heap across the end of the grid in a box that goes on: members beyond it
    are in the border cells however far they are, on every level."""
    sc = _box(700, 5 + levels, levels, dense=0.5)
    p, pos = sc["params"], sc["sub"]["pos"]
    mesh = 3 * sc["sub"]["radius"].max()
    a = "xyz"[axis]
    end = p["WorldOrigin_" + a] - mesh if side < 0 else p["WorldOrigin_" + a] + p["WorldSize_" + a] + mesh
    move = end - pos[:, axis].mean()
    for q in (pos, sc["clump"]["pos"]):
        q[:, axis] += move
    p["BoxLowLmt_" + a] -= 1.0
    p["BoxUpLmt_" + a] += 1.0
    _list(sc)
