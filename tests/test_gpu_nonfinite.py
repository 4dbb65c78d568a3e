"""What is not finite stays so in both components: in the lab frame the far
sums are real, but the reference forms them as complex products
(history_interaction.cpp:55-65), whose imaginary part is NaN where the real
one is not finite."""
import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I

pytestmark = pytest.mark.gpu

FORMS = [(p, m) for p in (capi.PREC_FP64, capi.PREC_MIXED) for m in (capi.COEF_TABLE, capi.COEF_ON_THE_FLY)]


@pytest.mark.parametrize("precision,mode", FORMS)
def test_lab_frame_field_at_a_whole_delay(golden_weights, precision, mode):
    c = I.Constants(c0=1.0, dt=0.125, num_timesteps=40, frame=1)
    dots = np.array([[0.0, 0, 0, 200, 10, 10, 0, 0, 2e-3],
                     [5.0, 0, 0, 200, 10, 10, 0, 0, 2e-3]])  # 40 steps
    hist = np.zeros((2, 40 + O.WINDOW, 2, 2), dtype=np.complex128)
    ref = O.history_evaluate(dots, c, *O.build_table(dots, c), hist, 39)
    assert np.isnan(ref.real).all() and np.isnan(ref.imag).all()
    with capi.Simulation(dots, I.make_pulse(), c, weights=golden_weights, precision=precision, coef_mode=mode) as sim:
        got = sim.history_evaluate(39)
    assert np.isnan(got.real).all() and np.isnan(got.imag).all()


@pytest.mark.parametrize("precision,mode", FORMS)
def test_lab_frame_field_of_an_infinite_sample(golden_weights, precision, mode):
    wl = I.plain_small(n=40, steps=200)
    c = wl.constants
    c.frame = 1
    hist = np.zeros((40, 200 + O.WINDOW, 2, 2), dtype=np.complex128)
    hist[7, :, 0, 1] = np.inf
    ref = O.history_evaluate(wl.dots, c, *O.build_table(wl.dots, c), hist, 180)
    bad = ~np.isfinite(ref.real)  # all but the dot itself and one whose window lies before step -22
    assert bad.sum() == 38 and np.isnan(ref.imag[bad]).all() and (ref[~bad] == 0).all()
    with capi.Simulation(wl.dots, wl.pulse, c, weights=golden_weights, precision=precision, coef_mode=mode) as sim:
        sim.set_history(-O.WINDOW, np.ascontiguousarray(hist[:, :, 0, 1].T))
        got = sim.history_evaluate(180)
    assert not np.isfinite(got.real[bad]).any() and np.isnan(got.imag[bad]).all()
    assert (got[~bad] == 0).all()
