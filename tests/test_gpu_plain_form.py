"""The far kernel's plain form in the blocks where some windows start before
step -22: it reads the samples of those steps as the zeros the ring was reset
to, and is taken only where that changes no bit.  Whatever the history holds
and whatever the coefficients, a run gives what it gives with "far_early" 0,
where each such sample is skipped."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from quest_b200 import capi, inputs as I

pytestmark = pytest.mark.gpu


def workload(n, frame, q, steps):
    wl = I.plain_table(seed=4, n=n, steps=steps, pulse_delay=0.05)
    wl.dots[:, 6:9] *= 0.1
    wl.constants.frame = frame
    wl.constants.interpolation_order = q
    return wl


@pytest.mark.parametrize("replay_before_reset", [False, True])
def test_a_replayed_evaluation_writes_the_ring(golden_weights, replay_before_reset):
    """qg_history_evaluate_noalloc captured once and replayed after a reset:
    its iterate goes into a slot that the first blocks' windows share with a
    step before -22, and the run is the one without it."""
    import torch

    wl = workload(300, 0, 5, 400)
    with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights, coef_mode=capi.COEF_TABLE) as sim:
        clean = sim.run(96)
        sim.set_option("reset", 1)
        step = sim.info()["ring_depth"] - 40  # step -40's slot
        assert 112 < step < 400
        d_in = torch.full((sim.n,), 1 + 1j, dtype=torch.complex128, device="cuda")
        d_out = torch.empty((sim.n,), dtype=torch.complex128, device="cuda")

        def evaluate(iterate, stream):
            rc = capi.lib().qg_history_evaluate_noalloc(
                sim.h, step, ctypes.c_void_p(d_in.data_ptr()) if iterate else None,
                ctypes.c_void_p(d_out.data_ptr()), ctypes.c_void_p(stream.cuda_stream))
            assert rc == capi.QG_OK, capi.lib().qg_last_error().decode()

        s = torch.cuda.Stream()
        evaluate(False, s)  # the first call looks the scratch's address up, before the capture
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            evaluate(True, torch.cuda.current_stream())
        if replay_before_reset:
            g.replay()
            torch.cuda.synchronize()
        sim.set_option("reset", 1)
        g.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(sim.get_history(step, 1)[0], np.full(sim.n, 1 + 1j))
        got = sim.run(96)
    np.testing.assert_array_equal(clean, got)


@pytest.mark.parametrize("precision,mode,scale", [
    (capi.PREC_FP64, capi.COEF_TABLE, 1e160), (capi.PREC_FP64, capi.COEF_ON_THE_FLY, 1e160),
    (capi.PREC_MIXED, capi.COEF_TABLE, 1e20), (capi.PREC_MIXED, capi.COEF_ON_THE_FLY, 1e20)])
@pytest.mark.parametrize("frame", [0, 1])
def test_coefficients_that_overflow(golden_weights, oracle_weights, precision, mode, scale, frame):
    """Dipoles whose coefficients are infinite in the precision they are held
    in: two dots 30.5 steps apart, no pulse.  Step 8 is the first with a tap
    that reads step -22, where the product with zero is NaN."""
    c = I.Constants(c0=1.0, dt=0.125, num_timesteps=40, frame=frame)
    dots = np.array([[0.0, 0, 0, 200, 10, 10, 0, 0, scale],
                     [30.5 * 0.125, 0, 0, 200, 10, 10, 0, 0, scale]])
    pulse = I.make_pulse(amplitude=0.0)
    if precision == capi.PREC_FP64:
        assert O.run_faithful(dots, pulse, c, oracle_weights, 40)[1] == 8
    for early in (1, 0):
        with capi.Simulation(dots, pulse, c, weights=golden_weights, precision=precision, coef_mode=mode) as sim:
            sim.set_option("far_early", early)
            with pytest.raises(capi.NonFiniteError) as e:
                sim.run(40)
        assert e.value.step == 8, early


@pytest.mark.parametrize("mode", [capi.COEF_TABLE, capi.COEF_ON_THE_FLY])
@pytest.mark.parametrize("precision", [capi.PREC_FP64, capi.PREC_MIXED])
@pytest.mark.parametrize("frame,q", [(0, 5), (1, 3)])
def test_both_forms_give_the_same_bits(golden_weights, mode, precision, frame, q):
    """All the blocks of a run from the ground state past the largest delay
    (about 300 steps), through a checkpoint taken among them."""
    wl = workload(700, frame, q, 352)
    outs = []
    for early in (1, 0):
        with capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights, precision=precision,
                             coef_mode=mode) as sim:
            sim.set_option("far_early", early)
            first = sim.run(40)
            data = sim.checkpoint()
            sim.run(24)
            sim.restore(data)
            outs.append(np.concatenate([first, sim.run(312)]))
    assert np.abs(outs[0][..., 1]).max() > 1e-8
    np.testing.assert_array_equal(outs[0], outs[1])


@pytest.mark.parametrize("precision,value", [(capi.PREC_FP64, 0.0), (capi.PREC_FP64, 1.0), (capi.PREC_FP64, np.nan),
                                             (capi.PREC_MIXED, 0.0), (capi.PREC_MIXED, 1.0)])
def test_a_checkpoint_brings_what_the_ring_holds(golden_weights, precision, value):
    """A checkpoint taken early, with an iterate written into a slot the next
    blocks' windows share with a step before -22: the loaded handle does not
    take the slot for a zero unless it is one, and continues as one that was
    never saved."""
    wl = workload(300, 0, 5, 400)

    def begin(early):
        sim = capi.Simulation(wl.dots, wl.pulse, wl.constants, weights=golden_weights, precision=precision,
                              coef_mode=capi.COEF_TABLE)
        sim.set_option("far_early", early)
        return sim

    outs = []
    for early in (1, 0):
        with begin(early) as a, begin(early) as b:
            a.run(32)
            step = a.info()["ring_depth"] - 40  # step -40's slot
            a.history_evaluate(step, np.full(a.n, value, dtype=np.complex128))
            b.restore(a.checkpoint())
            outs += [a.run(80), b.run(80)]
    for o in outs[1:]:
        np.testing.assert_array_equal(outs[0], o)
    assert np.isfinite(outs[0]).all()
