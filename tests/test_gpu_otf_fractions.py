"""On-the-fly coefficients at delays whose fraction is close to 0 or 1.

There the reference's Lagrange weights cancel (lagrange_set.cpp:17-41): a node
next to the fraction x has reciprocals of size 1/x, whose squares cancel in the
second derivative and leave its weight with an error of some
12 (3 q + 6) 2^-53 / x at the most, against a largest weight of 1 or more.
Both forms round those sums alike but not bit for bit, so one pair's field from
either agrees to the error the q + 1 taps then have on samples of size 3,
2 (q + 1) 12 (3 q + 6) 2^-53 3 / x, below 2e-12 / x for every order; half of
that is asked for."""
import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frame", [0, 1])
@pytest.mark.parametrize("q", [1, 3, 5, 7])
def test_fields_at_fractions_near_a_node(golden_weights, frame, q):
    c = I.Constants(num_timesteps=200, interpolation_order=q, frame=frame)
    rng = np.random.default_rng(q)
    hist = np.zeros((2, 200 + O.WINDOW, 2, 2), dtype=np.complex128)
    hist[:, :, 0, 1] = rng.uniform(-1, 1, (2, 222)) + 1j * rng.uniform(-1, 1, (2, 222))
    axis = np.array([0.48, 0.6, 0.64])
    for x in (1e-2, 1e-4, 1e-6):
        for delay in (16 + x, 17 - x, 83 + x, 84 - x):
            dots = np.array([[0.0, 0, 0, 200, 10, 10, 1e-3, 2e-3, -1e-3],
                             [*(axis * delay * 1e-3), 200, 10, 10, 2e-3, 1e-3, 1e-3]])
            ref = O.history_evaluate(dots, c, *O.build_table(dots, c), hist, 150)
            for mode in (capi.COEF_TABLE, capi.COEF_ON_THE_FLY):
                with capi.Simulation(dots, I.make_pulse(), c, weights=golden_weights, coef_mode=mode) as sim:
                    lo = max(-O.WINDOW, 151 - sim.info()["ring_depth"])
                    sim.set_history(lo, np.ascontiguousarray(hist[:, lo + O.WINDOW: 151 + O.WINDOW, 0, 1].T))
                    assert rel_err(ref, sim.history_evaluate(150)) <= 1e-12 / x, (delay, mode)
