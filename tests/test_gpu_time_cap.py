"""max_seconds holds within a chain of intervals too: a solve ends with the interval
that passes the cap, alone and in a batch, wherever the cap falls in a chain.

Bound: half of the caps, spread over more than a chain's length, are passed by less than
3 intervals (one, the error of the length a chain is given from the last one's time, and
the end of the solve); a chain that does not look is passed by half of its length."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N_GAS = 3.22e22
KT = 1.0 / (8.617333262e-5 * 300.0)
N = 8000000  # about 0.4 ms an interval: alone chains of 11, in a batch of 16


def _context(cap):
    from lokigpu import capi, synth
    ps = synth.flatten([synth.atomic_gas()])
    cfg = capi.default_config(n_electrons=float(N), n_interp=2000, seed=3, init_temp_ratio=KT, max_coll_before_ss=0.01,
                              req_integration_points=1e9, max_seconds=cap)
    ctx = capi.Context(cfg)
    ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
    ctx.set_conditions(N_GAS, 300.0, 100.0)
    return ctx


@pytest.mark.parametrize("batched", [False, True])
def test_time_cap_within_a_chain(batched):
    from lokigpu import capi
    over = []
    for k in range(12):
        cap = 0.15 + 0.9e-3 * k
        ctx = _context(cap)
        if batched:
            batch = capi.Batch(0, 1)
            batch.set_schedule(0)
            batch.add(ctx)
            (r,), status, _ = batch.run()
            assert status == [0]
            batch.close()
        else:
            r = ctx.solve()
        assert r.capped == 1 and r.elapsed > cap
        over.append((r.elapsed - cap) / (r.elapsed / r.sync_steps))
        ctx.close()
    assert np.median(over) <= 3.0, np.array(over)
