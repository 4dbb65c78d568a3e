"""The allocation-free evaluation adds the far terms in the order of the
regular one: the same bits for FP64 table handles with their own source
group."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,frame,q", [(2, 0, 5), (33, 1, 3), (200, 0, 5), (1000, 1, 5), (4096, 0, 4)])
def test_noalloc_gives_the_bits_of_history_evaluate(golden_weights, n, frame, q):
    import torch

    wl = I.plain_small(n=n, steps=400)
    wl.constants.frame = frame
    wl.constants.interpolation_order = q
    rng = np.random.default_rng(n)
    with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights, coef_mode=capi.COEF_TABLE) as sim:
        W = sim.info()["ring_depth"]
        hist = rng.normal(size=(W, n)) + 1j * rng.normal(size=(W, n))
        lo = max(-O.WINDOW, 380 - W + 1)
        sim.set_history(lo, hist)
        out = torch.empty((n,), dtype=torch.complex128, device="cuda")
        for step in (lo + W - 1, lo + W - 3):
            ref = sim.history_evaluate(step)
            rc = capi.lib().qg_history_evaluate_noalloc(sim.h, step, None, ctypes.c_void_p(out.data_ptr()), None)
            assert rc == capi.QG_OK, capi.lib().qg_last_error().decode()
            torch.cuda.synchronize()
            np.testing.assert_array_equal(ref, out.cpu().numpy())
