"""Engines of one process that step at the same time from several threads share
the GPU: their launches fit it together instead of taking turns."""
import threading
import time

import numpy as np
import pytest

import nbc
import scenegen as sg

pytestmark = pytest.mark.gpu


def _time(engines, steps):
    """Best of five: all of them stepped from threads of their own, three calls each."""
    def work(e):
        for _ in range(3):
            e.step(steps)
    best = np.inf
    for _ in range(5):
        ts = [threading.Thread(target=work, args=(e,)) for e in engines]
        t0 = time.perf_counter()
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        best = min(best, time.perf_counter() - t0)
    return best


def test_eight_engines_share_the_gpu():
    """Latency binds a scene of this size: eight side by side on an eighth of the
    SMs each take two to three times as long as one; in turns, six to eight."""
    scenes = [sg.make_test_tetra(n_clumps=2000, seed=s, intruder=None) for s in range(8)]
    for sc in scenes:   # at rest: no rebuild ends a launch
        sc["params"]["Gravity"] = 0.0
        sc["params"]["Thresh"] = 1.0
        sc["clump"]["vel"][:] = 0.0
        sc["clump"]["angvel"][:] = 0.0
    engines = [nbc.Engine([sc]) for sc in scenes]
    for e in engines:
        e.step(20)
    _time(engines, 20)   # (the launches for a share of the GPU are made on first use)
    one = _time(engines[:1], 100)
    assert _time(engines, 100) < 4.5 * one


def test_results_do_not_depend_on_the_neighbours():
    scenes = [sg.make_test_tetra(n_clumps=n, seed=n, intruder=None, thresh_ratio=0.02) for n in (30, 300, 900, 1700, 45)]
    alone = []
    for sc in scenes:
        e = nbc.Engine([sc])
        for _ in range(8):
            e.step(15)
        e.sync()
        alone.append((e.clumps(), e.pairs(), e.stats()))
    engines = [nbc.Engine([sc]) for sc in scenes]

    def work(e):
        for _ in range(8):
            e.step(15)
        e.sync()
    ts = [threading.Thread(target=work, args=(e,)) for e in engines]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for e, (c, p, st) in zip(engines, alone):
        d = e.clumps()
        for k in ("pos", "vel", "angvel", "quat", "force", "torque"):
            assert np.array_equal(c[k], d[k]), k
        assert all(np.array_equal(x, y) for x, y in zip(p, e.pairs())) and st == e.stats()
