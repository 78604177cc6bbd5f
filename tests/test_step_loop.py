"""Many steps in one launch (the default stepping) against one launch per pass
(eager), bitwise: scenes of a few warps, scenes with more work items than the
launch has warps, more scenes than the launch keeps in shared memory, step
limits reached inside a launch, and engines stepping at the same time from
several threads."""
import threading

import numpy as np
import pytest

import nbc
import scenegen as sg

pytestmark = pytest.mark.gpu

KEYS = ("pos", "vel", "angvel", "quat", "force", "torque")


def _same(a, b, s=0):
    ca, cb = a.clumps(s), b.clumps(s)
    for k in KEYS:
        assert np.array_equal(ca[k], cb[k]), (s, k)
    assert a.stats(s) == b.stats(s)
    assert a.contact_counts() == b.contact_counts()


def _scenes(kind):
    if kind == "one":
        return [sg.make_test_tetra(n_clumps=1, seed=3, intruder=None)]
    if kind == "small":
        return [sg.make_test_tetra(n_clumps=37, seed=4, intruder="sphere", wall="cube")]
    if kind == "spheres":   # a driver's behaviour, one-sphere clumps, the cylinder
        return [sg.as_sphere_driver(sg.make_test_spheres(n=333, seed=5, intruder=None, wall="cylinder"), "cylinder")]
    if kind == "large":     # more warps of clumps, pairs and boundary items than a launch has
        return [sg.make_test_tetra(n_clumps=11000, seed=6, intruder="cylinder", thresh_ratio=0.002)]
    few = [sg.make_test_tetra(n_clumps=2 + k % 3, seed=k, intruder=None) for k in range(6)]
    return [few[k * k % 6] for k in range(530)]


@pytest.mark.parametrize("precision", ["mixed", "f64"])
@pytest.mark.parametrize("kind", ["one", "small", "spheres", "large", "many"])
def test_loop_equals_eager(kind, precision):
    scenes = _scenes(kind)
    a = nbc.Engine(scenes, precision=precision, pair_slack=3.0)
    b = nbc.Engine(scenes, precision=precision, pair_slack=3.0, use_graph=False)
    assert a.launch_info()["step_loop"] == 1
    for n in (1, 2, 13, 8):
        a.step(n)
        b.step(n)
    a.sync()
    b.sync()
    for s in (0, len(scenes) // 2, len(scenes) - 1):
        _same(a, b, s)
        if scenes[s].get("intruder") is not None:
            assert np.array_equal(a.intruder_history(s, 24), b.intruder_history(s, 24))


def test_limits_inside_a_launch():
    scenes = _scenes("many")[:40]
    a = nbc.Engine(scenes, pair_slack=3.0)
    b = nbc.Engine(scenes, pair_slack=3.0, use_graph=False)
    for e in (a, b):
        for s in range(0, 40, 3):
            e.set_steps(5 + s, s)
        e.step(30)
        e.sync()
    for s in range(40):
        _same(a, b, s)


def test_engines_from_several_threads():
    scenes = [sg.make_test_tetra(n_clumps=n, seed=n, intruder=None) for n in (40, 700, 1500, 90)]
    alone = []
    for sc in scenes:
        e = nbc.Engine([sc])
        e.step(60)
        e.sync()
        alone.append(e.clumps())
    engines = [nbc.Engine([sc]) for sc in scenes]

    def work(e):
        for _ in range(6):
            e.step(10)
        e.sync()
    ts = [threading.Thread(target=work, args=(e,)) for e in engines]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for e, ref in zip(engines, alone):
        c = e.clumps()
        for k in KEYS:
            assert np.array_equal(c[k], ref[k]), k
