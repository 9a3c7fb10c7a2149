"""A job that arrives while another one runs, and a cancellation, do not wait for a
chain of intervals (up to 16): only for the intervals that are launched already, the
running one and at most one more.

An interval of the running job takes about half a millisecond, a chain eight. Bounds:
the median over arrivals spread over a chain, 4 intervals (two, and what the host needs
to admit or retire a job); without the rule it is half a chain."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N_GAS = 3.22e22
KT = 1.0 / (8.617333262e-5 * 300.0)


@pytest.fixture(scope="module")
def atomic():
    from lokigpu import synth
    return synth.flatten([synth.atomic_gas()])


def _submit(srv, ps, n, **kw):
    from lokigpu import capi
    cfg = capi.default_config(n_electrons=float(n), n_interp=2000, seed=3, init_temp_ratio=KT, max_coll_before_ss=0.01,
                              **kw)
    return srv.submit(cfg, ps, ps.gas_first, ps.gas_last, ps.gas_fraction, N_GAS, 300.0, 100.0)


def _interval(srv):
    a, t0 = srv.report().intervals, time.perf_counter()
    time.sleep(0.3)
    return (time.perf_counter() - t0) / (srv.report().intervals - a)


def test_arrivals_and_cancellations_wait_for_launched_intervals_only(atomic):
    from lokigpu import capi
    srv = capi.Server(0, 4)
    big = _submit(srv, atomic, 10000000, req_integration_points=1e9)
    while srv.report().intervals < 300:  # past the steady state and the tuning
        time.sleep(0.05)
    one = _interval(srv)
    waits, ends = [], []
    for k in range(15):
        time.sleep(0.02 + 0.6e-3 * k)
        jid = _submit(srv, atomic, 1000, max_sync_steps=1)
        st = srv.wait(jid, 60.0)
        assert st.state == capi.JOB_DONE
        waits.append(st.start_time - st.submit_time)
    for k in range(15):
        jid = _submit(srv, atomic, 1000, req_integration_points=1e9)
        while srv.poll(jid).state != capi.JOB_RUNNING:
            time.sleep(1e-3)
        time.sleep(0.02 + 0.6e-3 * k)
        t0 = time.perf_counter()
        srv.cancel(jid)
        assert srv.wait(jid, 60.0).state == capi.JOB_CANCELLED
        ends.append(time.perf_counter() - t0)
    srv.cancel(big)
    srv.wait(big, 60.0)
    srv.stop()
    assert np.median(waits) <= 4.0 * one, (np.array(waits) / one, one)
    assert np.median(ends) <= 4.0 * one, (np.array(ends) / one, one)
