"""Intervals that follow one another without a look by the host (run_chain) against
the same intervals one at a time, and the places where a chain has to end: caps,
samples every few intervals, error checks. The device's next control block is the
host's to the bit, so without ionization and attachment the series are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N_GAS = 3.22e22
KT = 1.0 / (8.617333262e-5 * 300.0)
F_AC = N_GAS * 1e-14 / (2 * np.pi)


def _context(n, angle=180.0, freq=0.0, mag=0.0, thermal=0, gas="atomic", **kw):
    from lokigpu import capi, synth
    ps = synth.flatten([synth.atomic_gas() if gas == "atomic" else synth.reid_ramp_gas()])
    cfg = capi.default_config(n_electrons=float(n), n_interp=2000, seed=31, init_temp_ratio=KT,
                              gas_temperature_effect=thermal, n_phases=8, **kw)
    ctx = capi.Context(cfg)
    ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
    ctx.set_conditions(N_GAS, 300.0, 100.0 if gas == "atomic" else 12.0, angle, freq, mag)
    return ctx


SERIES = [(0, 1), (1, 1), (2, 3), (3, 3), (4, 9), (5, 9), (6, 3), (7, 9)]


@pytest.mark.parametrize("n,kw", [(1, {}), (777, {}), (40000, {}), (5000, dict(freq=F_AC)),
                                  (5000, dict(angle=90.0, mag=500.0, thermal=1)), (3000, dict(gas="reid", thermal=2))])
def test_chained_intervals_repeat_single_ones(n, kw):
    a, b = _context(n, **kw), _context(n, **kw)
    a.init_ensemble()
    b.init_ensemble()
    ra = a.advance(75)
    for k in range(75):
        rb = b.advance(1)
    assert (ra.sync_steps, ra.time, ra.trial_freq) == (rb.sync_steps, rb.time, rb.trial_freq) and ra.sync_steps == 75
    assert (ra.real_collisions, ra.null_collisions, ra.max_energy) == (rb.real_collisions, rb.null_collisions, rb.max_energy)
    for which, width in SERIES:
        x, y = a.series(which, width), b.series(which, width)
        # sums over blocks in FP64: the order of their atomics moves the last bits
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-12 * np.abs(y).max())
    t = a.timing()
    assert t.advance_launches == 75 and t.electron_steps == 75.0 * n and t.advance_ms > 0
    a.close()
    b.close()


@pytest.mark.parametrize("kw", [dict(max_sync_steps=1), dict(max_sync_steps=150), dict(sync_oversampling=3),
                                dict(errors_checked=1, req_err_mean_energy=0.05), dict(max_coll_after_ss=60.0),
                                dict(req_ss_times=2.5), dict(req_integration_points=1.0)])
def test_a_chain_ends_where_the_host_decides(kw):
    from lokigpu import capi
    kw = dict(dict(req_integration_points=230.0, max_coll_before_ss=1e-6), **kw)
    alone, batched = _context(6001, **kw), _context(6001, **kw)
    r = alone.solve()
    batch = capi.Batch(0, 1)
    batch.add(batched)
    res, status, _ = batch.run()
    assert status == [0]
    q = res[0]
    for f in ("sync_steps", "integration_points", "sampling_points", "first_integration_index", "real_collisions",
              "null_collisions", "final_time", "ss_time", "capped", "trial_freq", "max_eedf_energy"):
        assert getattr(r, f) == getattr(q, f), f
    np.testing.assert_array_equal(alone.process_results()[0], batched.process_results()[0])
    np.testing.assert_array_equal(alone.distributions()["eedf"], batched.distributions()["eedf"])
    batch.close()
    alone.close()
    batched.close()
