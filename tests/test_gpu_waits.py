"""The step kernels' bounded waits: a launch in which nothing waits leaves no
trace of a block told not to post its steps."""
import numpy as np
import pytest

from quest_b200 import capi, inputs as I

pytestmark = pytest.mark.gpu


def test_posts_skipped_where_nothing_waits_are_forgotten(golden_weights):
    """Launches of two steps wait for no other block; a longer one does, and
    counts on what each block has posted so far."""
    wl = I.plain_small(n=200, steps=100, pulse_delay=0.05)
    wl.dots[:, 6:9] *= 0.1
    with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights) as sim:
        assert sim.info()["fused_step"] == 2
        ref = sim.run(66)
    with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights) as sim:
        sim.set_option("wait_limit", 20000)
        sim.set_option("test_skip_post", 3)
        got = [sim.run(2) for _ in range(3)]
        sim.set_option("test_skip_post", -1)
        got.append(sim.run(60))
    np.testing.assert_array_equal(ref, np.concatenate(got))
