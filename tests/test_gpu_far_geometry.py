"""The far kernels where a source's windows lie far apart (a line of dots
5 c dt apart) and close together (a tight cluster beside a line), through the
first blocks and the ring's wrap, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi
from tests.conftest import rel_err
from tests.test_gpu_parity import line_of_dots

pytestmark = pytest.mark.gpu

STEPS = 300


def workload(geometry):
    if geometry == "line":
        return line_of_dots(256, 5e-3)
    wl = line_of_dots(256, 4e-3)
    rng = np.random.default_rng(8)
    wl.dots[:128, 0:3] = rng.uniform(-0.01, 0.01, size=(128, 3))
    wl.dots[:128, 8] = 2e-5
    return wl


@pytest.mark.parametrize("geometry", ["line", "cluster_and_line"])
@pytest.mark.parametrize("mode", [capi.COEF_TABLE, capi.COEF_ON_THE_FLY])
def test_long_and_short_window_runs(golden_weights, oracle_weights, geometry, mode):
    wl = workload(geometry)
    hist, bad = O.run_fast(wl.dots, wl.pulse, wl.constants, oracle_weights, STEPS)
    assert bad is None
    ref = O.rho_trajectory(hist)
    assert np.abs(ref[..., 1]).max() > 1e-8
    for precision, bar in ((capi.PREC_FP64, 1e-10), (capi.PREC_MIXED, 1e-6)):
        with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights, precision=precision,
                             coef_mode=mode) as sim:
            got = sim.run(STEPS)
        for k in range(2):
            assert rel_err(ref[..., k], got[..., k]) <= bar
