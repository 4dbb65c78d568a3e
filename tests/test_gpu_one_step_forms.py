"""One-step FP64 evaluations at sizes on both sides of the lines between the
one-step far kernel's forms (table entries fetched three, two or one source
ahead, by how many of its blocks the device holds at once), against the
oracle's per-target sums, and through the allocation-free entry point with the
regular one's bits.

Both sums add n (q + 1) products in some order, so each is within
n (q + 1) 2^-53 (1 + small) of the exact one relative to the sum of the
products' sizes; their coefficients agree to a few ulp."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I

pytestmark = pytest.mark.gpu


def product_sizes(wl, targets):
    """sum over sources and taps of |coefficient| for each target (samples of
    size 1), from the closed form of the coefficients."""
    c = wl.constants
    q, dots = c.interpolation_order, wl.dots
    out = np.zeros(len(targets))
    for k, a in enumerate(targets):
        b = np.arange(len(dots)) != a
        dr = dots[a, :3] - dots[b, :3]
        r = np.linalg.norm(dr, axis=1)
        x = r / (c.c0 * c.dt) % 1.0
        dd = dots[b, 6:] @ dots[a, 6:]
        ab = (dots[b, 6:] * dr).sum(1) * (dr @ dots[a, 6:]) / r**2
        G0, G1, G2 = (dd - 3 * ab) * c.c0**2 / r**3, (dd - 3 * ab) * c.c0 / r**2, (dd - ab) / r
        om = c.laser_frequency if c.frame == 0 else 0.0
        for i in range(q + 1):
            p = np.poly1d([m for m in range(q + 1) if m != i], r=True)
            p = p / p(i)
            w0, w1, w2 = p(x), -p.deriv()(x) / c.dt, p.deriv(2)(x) / c.dt**2
            tap = G0 * w0 + G1 * (w1 + 1j * om * w0) + G2 * (w2 + 2j * om * w1 - om**2 * w0)
            out[k] += np.abs(tap).sum() * c.mu0 / (4 * np.pi * c.hbar) * (2 if c.frame else 1)
    return out


@pytest.mark.parametrize("n,q", [(1500, 5), (2047, 4), (2500, 7), (3500, 5), (4090, 5), (5200, 3)])
@pytest.mark.parametrize("frame", [0, 1])
def test_one_step_forms_against_oracle(golden_weights, n, q, frame):
    import torch

    wl = I.plain_table(seed=5, n=n, steps=900)
    c = wl.constants
    c.frame, c.interpolation_order = frame, q
    rng = np.random.default_rng(n)
    with capi.Simulation(wl.dots, wl.pulse, c, weights=golden_weights, coef_mode=capi.COEF_TABLE) as sim:
        W = sim.info()["ring_depth"]
        step = 700
        lo = step - W + 1
        t = np.arange(lo, step + 1)[:, None]
        hist = np.exp(1j * (rng.uniform(0, 6, n) + 0.01 * rng.uniform(-1, 1, n) * t))
        sim.set_history(lo, hist)
        got = sim.history_evaluate(step)
        if n <= 4096:
            out = torch.empty((n,), dtype=torch.complex128, device="cuda")
            rc = capi.lib().qg_history_evaluate_noalloc(sim.h, step, None, ctypes.c_void_p(out.data_ptr()), None)
            assert rc == capi.QG_OK, capi.lib().qg_last_error().decode()
            torch.cuda.synchronize()
            np.testing.assert_array_equal(got, out.cpu().numpy())
    targets = np.sort(rng.choice(n, size=48, replace=False))
    ref = O.history_evaluate_targets(wl.dots, c, np.ascontiguousarray(hist.T), lo, step, targets)
    bound = 2 * (n * (q + 1) + 64) * 2.0**-53 * product_sizes(wl, targets)
    assert np.abs(ref).max() > 1e3 * bound.max()
    assert (np.abs(got[targets] - ref) <= bound).all()
