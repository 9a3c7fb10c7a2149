"""The advance of a condition on its own where its launch changes: two, three and four
blocks per SM (77,824 and 116,736 electrons on 152 SMs), under DC and crossed B.
Without ionization and attachment no result depends on the launch: collision counts
equal those of the batched solve, whose warps take chunks from a counter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N_GAS = 3.22e22


@pytest.mark.parametrize("n,mag,thermal", [
    (77823, 0.0, 0), (77824, 0.0, 2), (77825, 0.0, 0), (116735, 0.0, 1), (116736, 0.0, 0),
    (116737, 0.0, 0), (77824, 500.0, 0), (116736, 500.0, 1), (116737, 500.0, 0)])
def test_launch_changes(n, mag, thermal):
    from lokigpu import capi, synth
    ps = synth.flatten([synth.atomic_gas()])

    def context():
        cfg = capi.default_config(n_electrons=float(n), n_interp=2000, seed=78, init_temp_ratio=40.0,
                                  gas_temperature_effect=thermal, max_coll_before_ss=1e-6, req_integration_points=60.0)
        ctx = capi.Context(cfg)
        ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
        ctx.set_conditions(N_GAS, 300.0, 100.0, 90.0 if mag else 180.0, 0.0, mag)
        return ctx

    alone, batched = context(), context()
    a = alone.solve()
    batch = capi.Batch(0, 1)
    batch.add(batched)
    res, status, _ = batch.run()
    assert status == [0]
    assert (a.real_collisions, a.null_collisions) == (res[0].real_collisions, res[0].null_collisions)
    np.testing.assert_array_equal(alone.process_results()[0], batched.process_results()[0])
    batch.close()
    alone.close()
    batched.close()
