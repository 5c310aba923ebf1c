"""Failure detection on the GPU without a fault.

Every device-side wait in the library is bounded: the onesweep sort's
decoupled look-back gives up after a fixed number of polls of an empty status
word, sets an error bit and lets the kernel finish; the host reads the bit and
returns JT_ETIMEDOUT.  jt_wait_probe runs that same wait on a status word
that nothing publishes.  The test checks that it times out, reports it, and
that the context still computes forces afterwards.
"""
import ctypes as C

import numpy as np
import pytest

import janus_treepm as J

pytestmark = pytest.mark.gpu


def test_bounded_wait_times_out_and_reports():
    flag = C.c_int(-1)
    rc = J.library().jt_wait_probe(1 << 16, C.byref(flag))
    assert rc == J.JT_ETIMEDOUT and flag.value == 1
    # the context is intact: a force evaluation still works
    rng = np.random.default_rng(1)
    pp = rng.uniform(-16, 16, (2000, 3)).astype(np.float32)
    pm = rng.uniform(-16, 16, (2000, 3)).astype(np.float32)
    s = J.Solver(J.Config(box_L=32.0, pm_grid=32, softening=0.05))
    s.set_state(pp, None, pm, None)
    ap, am = s.accel()
    assert np.all(np.isfinite(ap)) and np.all(np.isfinite(am))
    s.close()


def test_probe_rejects_bad_limits():
    flag = C.c_int()
    assert J.library().jt_wait_probe(0, C.byref(flag)) == J.JT_EINVAL
    assert J.library().jt_wait_probe(1 << 25, C.byref(flag)) == J.JT_EINVAL


@pytest.mark.parametrize("code", [J.JT_EOVERFLOW, J.JT_ETIMEDOUT])
def test_device_error_ends_a_call_of_many_steps(code):
    """The error word is set before the call: the step that meets it and at most
    one more run (drifts of dt v show how many), the call reports the error, and
    the next call works."""
    n, dt, v = 300, 0.25, 0.125
    rng = np.random.default_rng(2)
    pp = rng.uniform(-16, 0, (n, 3)).astype(np.float32)
    vp = np.full((n, 3), v, np.float32)
    s = J.Solver(J.Config(box_L=32.0, pm_grid=32, softening=0.05, G_mass_plus=1e-12))
    s.set_state(pp, vp, pp[:0], vp[:0])
    s.accel()
    assert J.library().jt_inject_error(s._h, code) == J.JT_OK
    with pytest.raises(J.JanusError) as e:
        s.step(dt, 0.0, 1.0, 12)
    assert e.value.code == code
    steps = (s.get_state()[0] - pp) / (dt * v)
    assert 0.99 < steps.min() and steps.max() < 2.01, (steps.min(), steps.max())
    s.step(dt, 0.0, 1.0, 3)
    steps2 = (s.get_state()[0] - pp) / (dt * v) - steps
    assert np.abs(steps2 - 3).max() < 0.01
    assert J.library().jt_inject_error(s._h, J.JT_EBUSY) == J.JT_EINVAL
    s.close()


def test_failed_host_step_leaves_nothing_for_the_next_call():
    """A round trip whose force pass fails on the host: its kick and drift are
    not in the next call's timings, and the round trip works again."""
    rng = np.random.default_rng(3)
    pp = rng.uniform(-15, 15, (900, 3)).astype(np.float32)
    pm = rng.uniform(-15, 15, (800, 3)).astype(np.float32)
    s = J.Solver(J.Config(box_L=32.0, pm_grid=32, softening=0.05))
    s.set_state(pp, None, pm, None)
    ap, am = s.accel()
    state = [pp.copy(), np.zeros_like(pp), ap.copy(), pm.copy(), np.zeros_like(pm), am.copy()]
    assert J.library().jt_inject_error(s._h, J.JT_ECUDA) == J.JT_OK
    with pytest.raises(J.JanusError) as e:
        s.step_host(*[a.copy() for a in state], 1e-3, 0.0, 1.0)
    assert e.value.code == J.JT_ECUDA
    s.accel()
    assert s.timings()["kick_drift_ms"] == 0.0
    s.step_host(*state, 1e-3, 0.0, 1.0)
    t = s.timings()
    assert 0.0 < t["kick_drift_ms"] < t["total_ms"]
    s.set_state(pp, None, pm, None)
    s.step(1e-3, 0.0, 1.0, 1)
    assert np.abs(s.get_state()[0] - state[0]).max() < 1e-5
    s.close()
