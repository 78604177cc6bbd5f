"""The launch shapes on the path that reads them: blocks per SM of the pair
kernel in steps of one launch per pass, and the tuner's trials on the path its
options ask for."""
import os

import numpy as np
import pytest

import nbc
import scenegen as sg

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def test_pair_blocks_give_the_same_results():
    """A settled bed with more near pairs than the smallest grid has threads
    (148 SMs x 2 blocks x 256), so that the grids differ and the smallest walks
    its items several times."""
    sc = sg.tetra_state_from_npz(os.path.join(GOLDEN, "cfg1_settled.npz"))
    ref = None
    for blocks in (2, 5, 16):
        e = nbc.Engine([sc], precision="mixed", use_graph=False, pair_blocks=blocks)
        assert e.launch_info() == {"step_loop": 0, "search_lanes": 8, "clump_batch": 1, "pair_blocks": blocks}
        e.step(10)
        e.sync()
        assert e.contact_counts()[0] > 2 * 148 * 2 * 256
        out = (e.clumps(), e.pairs(), e.stats())
        e.close()
        ref = ref or out
        for k in ("pos", "vel", "angvel", "quat", "force", "torque"):
            assert np.array_equal(out[0][k], ref[0][k]), (blocks, k)
        assert np.array_equal(out[1], ref[1]) and out[2] == ref[2]


def test_reported_shapes_are_those_in_use():
    sc = sg.make_test_tetra(n_clumps=20, seed=1, intruder=None)
    e = nbc.Engine([sc], search_lanes=32, clump_batch=4, pair_blocks=4)
    assert e.launch_info() == {"step_loop": 1, "search_lanes": 8, "clump_batch": 1, "pair_blocks": 4}


def test_tuner_times_the_path_of_its_options():
    """One launch per pass takes a scene of this size over twice as long a step as the
    loop of steps on the device, which has no pair kernel to tune."""
    sc = sg.make_test_tetra(n_clumps=150, seed=2, intruder=None)
    loop = nbc.autotune([sc], trial_steps=100)
    assert loop["pair_blocks"] == 12
    eager = nbc.autotune([sc], trial_steps=100, use_graph=False)
    assert eager["pair_blocks"] in (4, 8, 12, 16)
    assert eager["ms_per_step"] > 1.5 * loop["ms_per_step"]
