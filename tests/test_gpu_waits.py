"""The step kernels' bounded waits: a launch in which nothing waits leaves no
trace of a block told not to post its steps, and the general form's exchange
between the blocks of its grid ends with an error that the host reads when one
of them never arrives."""
import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I
from tests.conftest import rel_err
from tests.test_gpu_group_step import cloud

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


def test_exchange_that_runs_out_returns_an_error_and_the_handle_recovers(golden_weights, oracle_weights):
    dots, pulse, c = cloud(400, 32)  # a grid of blocks: more rows than one cluster's warps
    with capi.Simulation(dots, pulse, c, weights=golden_weights) as sim:
        assert sim.info()["fused_step"] == 0
        sim.set_option("wait_limit", 2000)
        sim.set_option("test_skip_post", 1)
        with pytest.raises(capi.QuestError) as e:
            sim.run(20, record=False)
        assert e.value.code == capi.QG_ERR_CUDA and "timed out" in str(e.value)
        sim.set_option("test_skip_post", -1)
        sim.set_option("wait_limit", 0)
        sim.set_option("reset", 1)
        got = sim.run(32)
    hist, bad = O.run_fast(dots, pulse, c, oracle_weights, 32)
    assert bad is None
    ref = O.rho_trajectory(hist)
    for k in range(2):
        assert rel_err(ref[..., k], got[..., k]) <= 1e-10  # the FP64 path's bar
