"""The far kernel cuts its source groups into parts so that small ensembles
fill the device, and skips the sources whose windows lie before step -22.  At
sizes and groups where the cut leaves short, empty or ragged parts, runs from
the ground state through the first blocks agree with the oracle (FP64, table
and on the fly, both frames), and mixed precision with FP64."""
import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu

STEPS = 150


def workload(n, frame, q):
    wl = I.plain_small(n=n, steps=STEPS, pulse_delay=0.03)
    wl.dots[:, 8] = 2e-4
    wl.constants.frame = frame
    wl.constants.interpolation_order = q
    return wl


def run(wl, weights, group=None, **kw):
    with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=weights, **kw) as sim:
        if group is not None:
            sim.set_option("far_group", group)
        return sim.run(STEPS)


@pytest.mark.parametrize("n,frame,q", [(33, 0, 5), (161, 1, 3), (700, 0, 4), (700, 1, 7)])
def test_parts_of_every_group_against_oracle(golden_weights, oracle_weights, n, frame, q):
    # FP64 parity bar of the GPU path: 1e-10 of the largest value
    wl = workload(n, frame, q)
    hist, bad = O.run_fast(wl.dots, wl.pulse, wl.constants, oracle_weights, STEPS)
    assert bad is None
    ref = O.rho_trajectory(hist)
    runs = [run(wl, golden_weights, g, coef_mode=capi.COEF_TABLE) for g in (None, 1, 3, 5, 1000)]
    runs.append(run(wl, golden_weights, coef_mode=capi.COEF_ON_THE_FLY))
    for got in runs:
        for k in range(2):
            assert rel_err(ref[..., k], got[..., k]) <= 1e-10
    # the mixed form's bar against FP64: 1e-6
    for mode in (capi.COEF_TABLE, capi.COEF_ON_THE_FLY):
        mixed = run(wl, golden_weights, coef_mode=mode, precision=capi.PREC_MIXED)
        for k in range(2):
            assert rel_err(ref[..., k], mixed[..., k]) <= 1e-6


@pytest.mark.parametrize("mode,frame", [(capi.COEF_TABLE, 0), (capi.COEF_TABLE, 1), (capi.COEF_ON_THE_FLY, 0),
                                        (capi.COEF_ON_THE_FLY, 1)])
def test_one_step_evaluation_at_the_first_live_samples(golden_weights, mode, frame):
    """An evaluation sums one step: windows wholly before step -22 are
    skipped, those that reach it are cut at it."""
    wl = workload(130, frame, 5)
    c = wl.constants
    rng = np.random.default_rng(7)
    hist = np.zeros((wl.n, STEPS + O.WINDOW, 2, 2), dtype=np.complex128)
    hist[:, :, 0, 1] = rng.normal(size=(wl.n, STEPS + O.WINDOW)) + 1j * rng.normal(size=(wl.n, STEPS + O.WINDOW))
    delays, coefs = O.build_table(wl.dots, c)
    with capi.Simulation(wl.dots, wl.pulse, c, weights=golden_weights, coef_mode=mode) as sim:
        sim.set_history(-O.WINDOW, np.ascontiguousarray(hist[:, :, 0, 1].T))
        for step in (0, 1, 17, 100, STEPS - 1):
            ref = O.history_evaluate(wl.dots, c, delays, coefs, hist, step)
            assert rel_err(ref, sim.history_evaluate(step)) < 1e-12, step
