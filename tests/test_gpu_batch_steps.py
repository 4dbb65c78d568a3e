"""The step launches of a batch may start before the step before them has
ended; every block then waits for it.  Each member keeps the bits it has
alone: in batches of one block, of uneven members that end at different steps
and of more blocks than the device holds at once, in the block's graph and in
single launches."""
import numpy as np
import pytest

from quest_b200 import capi

from tests.test_gpu_batch import ensemble, solo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes, steps", [((5,), (48,)), ((33, 2, 400), (64, 32, 48)), ((1000,) * 20, (48,) * 20)],
                         ids=["one_block", "uneven", "more_blocks_than_fit"])
@pytest.mark.parametrize("single_launches", [0, 1])
def test_overlapping_step_launches_keep_the_order(golden_weights, sizes, steps, single_launches):
    ens = [ensemble(70 + i, n, 0.02 * n ** (1 / 3), s, 5.0 + i) for i, (n, s) in enumerate(zip(sizes, steps))]
    batch = capi.Batch(len(ens))
    batch.set_option("profile", single_launches)
    sims = [capi.Simulation(*e, weights=golden_weights) for e in ens]
    for s in sims:
        batch.add(s)
    batch.run(4)
    for i in sorted({0, len(ens) // 2, len(ens) - 1}):
        np.testing.assert_array_equal(sims[i].state(), solo(*ens[i], golden_weights, steps[i])[0])
    batch.close()
    for s in sims:
        s.close()


def test_member_ending_within_a_block_keeps_its_state(golden_weights):
    """Blocks run after such a member's last step change nothing of it."""
    ens = [ensemble(80 + i, 200, 0.1, s, 5.0) for i, s in enumerate((64, 17, 24, 40))]
    batch = capi.Batch(len(ens))
    sims = [capi.Simulation(*e, weights=golden_weights) for e in ens]
    for s in sims:
        batch.add(s)
    batch.run(4)
    for sim, e in zip(sims, ens):
        steps = e[2].num_timesteps
        assert sim.next_step == steps
        np.testing.assert_array_equal(sim.state(), solo(*e, golden_weights, steps)[0])
    batch.close()
    for s in sims:
        s.close()
