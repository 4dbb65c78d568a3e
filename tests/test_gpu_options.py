"""Options that name a form of the far launch are accepted in their ranges,
read back as set, and keep the batch's timing run off, as an explicit choice
does for a handle."""
import numpy as np
import pytest

from quest_b200 import capi, inputs as I

pytestmark = pytest.mark.gpu


def test_options_read_back(golden_weights):
    wl = I.plain_small(n=64, steps=32)
    with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights) as sim:
        for v in range(12):
            sim.set_option("far_variant", v)
            assert sim.get_option("far_variant") == v
        for v in (-1, 12):
            with pytest.raises(capi.QuestError):
                sim.set_option("far_variant", v)


@pytest.mark.parametrize("key", [None, "far_packed", "far_gmajor"])
def test_an_explicit_batch_choice_keeps_the_tuner_off(golden_weights, key):
    wl = I.plain_small(n=600, steps=64, pulse_delay=0.02)
    batch = capi.Batch(1)
    with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights) as sim:
        batch.add(sim)
        if key:
            for v in (1, 0):
                batch.set_option(key, v)
                assert batch.get_option(key) == v
        batch.run(1)
        assert (batch.get_option("tuned_far_us") > 0) == (key is None)
        batch.set_option("autotune", 1)
        batch.run(1)
        assert batch.get_option("tuned_far_us") > 0
        batch.close()
