"""Launches of the many-steps kernel are bounded, so that other streams of the
process get the GPU between two of them however long a call is; where they
begin and end changes no result."""
import numpy as np
import pytest

import nbc
import scenegen as sg

pytestmark = pytest.mark.gpu


def _launches(e, steps):
    e.timing_enable(0)
    e.step(steps)
    return e.timing_read()["kernel_launches"]


def test_long_calls_are_cut_into_launches():
    """A scene at rest never rebuilds its list: 1,000 steps were one launch."""
    sc = sg.make_test_tetra(n_clumps=300, seed=8, intruder=None)
    sc["params"]["Gravity"] = 0.0
    sc["params"]["Thresh"] = 1.0
    sc["clump"]["vel"][:] = 0.0
    sc["clump"]["angvel"][:] = 0.0
    e = nbc.Engine([sc])
    e.step(2)
    assert e.launch_info()["step_loop"] == 1
    assert _launches(e, 1000) >= 1 + 1000 // 128
    assert e.stats()["rebuilds"] == 1


@pytest.mark.parametrize("precision", ["mixed", "f64"])
def test_turns_change_nothing(precision):
    """Calls that end before, at and behind the end of a launch, with rebuilds
    at other steps, against one launch per pass."""
    sc = sg.make_test_tetra(n_clumps=60, seed=9, intruder="sphere", wall="cube", thresh_ratio=0.02)
    a = nbc.Engine([sc], precision=precision, pair_slack=3.0)
    b = nbc.Engine([sc], precision=precision, pair_slack=3.0, use_graph=False)
    for n in (1, 127, 128, 129, 300):
        a.step(n)
        b.step(n)
        a.sync()
        b.sync()
        ca, cb = a.clumps(), b.clumps()
        for k in ("pos", "vel", "angvel", "quat", "force", "torque"):
            assert np.array_equal(ca[k], cb[k]), (n, k)
        assert a.stats() == b.stats()
    assert a.stats()["rebuilds"] >= 2
