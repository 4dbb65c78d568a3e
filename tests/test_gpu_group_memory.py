"""The general step form where its shared memory does not hold everything:
near lists read from global memory (a dense group of 700 dots or more),
iterates (from about 13 600 dots) and rows' states (from about 214 000) left
there too, against the oracle.  The large ensembles are a coupled chain and its
retarded neighbours among dots without a dipole, which take part in every list
and exchange and change nothing."""
import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I
from tests.conftest import rel_err
from tests.test_gpu_group_step import check, cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [720, 1000])
def test_near_lists_in_global_memory(golden_weights, oracle_weights, n):
    check(*cloud(n, 36), golden_weights, oracle_weights, 36)


@pytest.mark.parametrize("bystanders", [12800, 14000, 216000])
def test_iterates_and_states_in_global_memory(golden_weights, oracle_weights, bystanders):
    steps = 20
    wl = I.plain_small(n=140, steps=steps, pulse_delay=0.01)
    wl.dots[:, 8] = 2e-5
    rng = np.random.default_rng(3)
    step = rng.normal(size=(40, 3))
    step *= 8e-4 / np.linalg.norm(step, axis=1, keepdims=True)
    step[:, 0] = np.abs(step[:, 0])
    wl.dots[:40, :3] = np.cumsum(step, 0)
    hist, bad = O.run_fast(wl.dots, wl.pulse, wl.constants, oracle_weights, steps)
    assert bad is None
    ref = O.rho_trajectory(hist)
    # a jittered grid 17.3 c dt apart: no two of its dots are within 16 steps
    m = int(np.ceil(bystanders ** (1 / 3)))
    at = np.arange(bystanders)
    far = np.zeros((bystanders, 9))
    far[:, :3] = (np.stack([at // (m * m), at // m % m, at % m], 1) - 0.5 * m) * 0.0173
    far[:, :3] += rng.uniform(-2e-4, 2e-4, size=(bystanders, 3))
    far[:, 3:6] = 200.0, 10.0, 10.0
    dots = np.concatenate([wl.dots, far])
    with capi.Simulation(dots, wl.pulse, wl.constants, weights=golden_weights,
                         coef_mode=capi.COEF_ON_THE_FLY) as sim:
        assert sim.info()["fused_step"] == 0
        sim.run(steps - 1, record=False)
        got = sim.run(1)[0, :140]
    for k in range(2):
        assert rel_err(ref[-1, :, k], got[:, k]) <= 1e-10  # the FP64 path's bar
    assert np.abs(ref[-1, :, 1]).max() > 1e-8
