"""The general step form (a group of dots coupled at delay 0 larger than a
32-dot block): one thread-block cluster while its near lists fit in shared
memory, a cooperative grid beyond, against the oracle, at sizes around a
block's rows and around the change of form, and for a coupled group among
dots that are not."""
import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


def cloud(n, steps, order=3):
    """n dots on a jittered grid, all within c dt of each other (the reference
    example's units and pulse, moved to arrive early)."""
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1 / 3)))
    at = rng.permutation(m ** 3)[:n]
    grid = np.stack([at // (m * m), at // m % m, at % m], 1)
    dots = np.empty((n, 9))
    dots[:, :3] = ((grid + 0.5 + 0.25 * (rng.random((n, 3)) - 0.5)) / m - 0.5) * 0.2
    dots[:, 3:6] = 2278.9013, 10.0, 20.0
    dots[:, 6:] = 5.2917721e-4, 0.0, 0.0
    pulse = I.make_pulse(15589.2260227, 0.15, 227.89013, 2278.9013, (0.0, 0.0, 7.6015964), (1.0, 0.0, 0.0))
    c = I.Constants(299.792458, 0.65821193, 2.0133545e-4, 2278.9013, 0.5e-2, order, steps, 0)
    return dots, pulse, c


def check(dots, pulse, c, weights, oracle_weights, steps, pieces=None):
    hist, bad = O.run_fast(dots, pulse, c, oracle_weights, steps)
    assert bad is None
    ref = O.rho_trajectory(hist)
    with capi.Simulation(dots, pulse, c, weights=weights) as sim:
        assert sim.info()["fused_step"] == 0
        got = np.concatenate([sim.run(k) for k in (pieces or [steps])])
    for k in range(2):
        assert rel_err(ref[..., k], got[..., k]) <= 1e-10  # the FP64 path's bar
    assert np.abs(ref[..., 1]).max() > 1e-4


@pytest.mark.parametrize("n", [33, 64, 257, 400, 497, 640])
def test_every_pair_coupled(golden_weights, oracle_weights, n):
    check(*cloud(n, 60), golden_weights, oracle_weights, 60)


def test_pieces_off_the_block_boundary(golden_weights, oracle_weights):
    check(*cloud(100, 70, order=5), golden_weights, oracle_weights, 70, pieces=[1, 20, 11, 38])


def test_a_coupled_chain_among_retarded_dots(golden_weights, oracle_weights):
    """40 dots in a chain closer than c dt, 1100 further ones: a sparse near
    list, far and mid pairs beside it, more rows than one cluster's warps."""
    wl = I.plain_small(n=1140, steps=80, pulse_delay=0.02)
    wl.dots[:, 8] = 2e-5
    rng = np.random.default_rng(3)
    step = rng.normal(size=(40, 3))
    step *= 8e-4 / np.linalg.norm(step, axis=1, keepdims=True)
    step[:, 0] = np.abs(step[:, 0])
    wl.dots[:40, :3] = np.cumsum(step, 0)
    hist, bad = O.run_fast(wl.dots, wl.pulse, wl.constants, oracle_weights, 80)
    assert bad is None
    ref = O.rho_trajectory(hist)
    with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights) as sim:
        assert sim.info()["fused_step"] == 0
        got = sim.run(80)
    for k in range(2):
        assert rel_err(ref[..., k], got[..., k]) <= 1e-10
