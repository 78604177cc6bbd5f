"""The clump pass's lane table: clumps of sizes at the edges of a warp's 32
lanes (none, one, 31, 32, 33, 64, 65 members, and sizes that leave idle lanes
between them) against the FP64 oracle, alone and as the second scene of a
batch; the caller's clump order is kept whatever order the engine uses."""
import numpy as np
import pytest

import nbc
import oracle
import scenegen as sg

pytestmark = pytest.mark.gpu


def _scene(sizes, seed, r=0.4e-3, steps=12):
    """Clumps of the given member counts, rotating and pressed into the floor
    and into one another along x; a small Thresh rebuilds the list often."""
    rng = np.random.default_rng(seed)
    rho, K = sg.MATERIAL["rho"], len(sizes)
    locals_, radii, masses, props, pos = [], [], [], [], []
    x = 0.0
    for n in sizes:
        d = rng.normal(size=(n, 3))
        d /= np.maximum(np.linalg.norm(d, axis=1), 1e-9)[:, None]
        R = r * max(1.0, n) ** (1 / 3)
        loc = d * R * rng.uniform(0.3, 1.0, (n, 1))
        rad = r * rng.uniform(0.8, 1.2, n)
        M = rho * 4 / 3 * np.pi * r ** 3 * max(n, 1)
        locals_.append(loc)
        radii.append(rad)
        masses.append(np.full(n, M / max(n, 1)))
        props.append([0.4 * M * (R + r) ** 2 * c for c in (1.0, 1.1, 1.2)] + [M])
        low = (loc[:, 2] - rad).min() if n else 0.0
        x += R + r
        pos.append([x, 0.0, -low - 0.02 * r])
        x += R + 0.9 * r
    pos = np.array(pos)
    params = sg.default_params(StepSize=2e-7, EndStep=steps, OutputInterval=1, Thresh=3e-4 * r, BranchLmtLen=256)
    hi = np.array([x + 5 * r, 20 * r, 40 * r])
    sg.set_world_box(params, [-5 * r, -20 * r, -2 * r], hi)
    return sg.assemble(params, pos, np.tile([0, 0, 0, 1.0], (K, 1)), rng.uniform(-0.3, 0.3, (K, 3)),
                       rng.uniform(-150, 150, (K, 3)), np.array(props), locals_, radii, masses,
                       cube=sg.make_cube((x + 50 * r, 100 * r, 50 * r), (0.0, 0.0, 50 * r)))


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("sizes", [[33], [32, 1, 31, 0, 2], [5, 0, 64, 27, 6, 65, 1, 1, 33, 30, 3], [1] * 33 + [8] * 5])
def test_clump_sizes_against_oracle(sizes):
    sc = _scene(sizes, seed=len(sizes))
    o = oracle.OracleScene(sc)
    o.step(12)
    co = o.clumps()
    first = sg.make_test_tetra(n_clumps=11, seed=3, intruder=None)
    alone = nbc.Engine([sc], precision="f64")
    both = nbc.Engine([first, sc], precision="f64")
    for e, s in ((alone, 0), (both, 1)):
        e.step(12)
        e.sync()
        ce = e.clumps(s)
        # positions to rounding; velocities by the forces' rounding over the overlap (1e-16 R / 1e-2 r a step)
        for k, tol in (("pos", 1e-12), ("quat", 1e-12), ("vel", 1e-9), ("angvel", 1e-9)):
            assert _rel(ce[k], co[k]) < tol, (k, _rel(ce[k], co[k]))
        assert np.array_equal(e.subspheres(s)["clump_id"], o.sub()["clump_id"])
        assert e.stats(s)["rebuilds"] >= 2
    for k in ("pos", "vel", "quat", "angvel", "force", "torque"):
        assert np.array_equal(alone.clumps(0)[k], both.clumps(1)[k]), k
