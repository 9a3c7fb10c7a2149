"""The distributions a context on its own counts with the moments of each sample
(k_sample) against the same condition in a batch, which counts them in separate
passes below 150,000 electrons and with its samples in other chunks above: without ionization and attachment both see the same electrons, so every
count, and with it every reported value, is equal. Sizes around a warp, a block,
the change of the block size and of the EVDF's place, odd grids and grids too
large for shared memory, in one direction or both; small ensembles re-bin often,
which leaves a sample to the separate passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N_GAS = 3.22e22
DEFAULT = (1000, 100, 200, 200)


def _context(n, cells, freq, thermal):
    from lokigpu import capi, synth
    ps = synth.flatten([synth.atomic_gas()])
    cfg = capi.default_config(n_electrons=float(n), n_interp=2000, seed=77, init_temp_ratio=1.0 / (8.617333262e-5 * 300.0),
                              gas_temperature_effect=thermal, max_coll_before_ss=1e-6, req_integration_points=60.0,
                              n_energy_cells=cells[0], n_cos_cells=cells[1], n_radial_cells=cells[2],
                              n_axial_cells=cells[3], n_phases=8)
    ctx = capi.Context(cfg)
    ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
    ctx.set_conditions(N_GAS, 300.0, 100.0, 180.0, freq, 0.0)
    return ctx


@pytest.mark.parametrize("n,cells,freq,thermal", [
    (1, DEFAULT, 0.0, 0), (33, DEFAULT, 0.0, 0), (511, (4096, 3, 33, 31), 0.0, 2), (20000, (17, 100, 400, 400), 0.0, 0),
    (77823, DEFAULT, 0.0, 0), (77825, DEFAULT, N_GAS * 1e-14 / (2 * np.pi), 0), (999999, DEFAULT, 0.0, 0),
    (1000001, (999, 99, 199, 201), 0.0, 0), (1000001, (17, 100, 400, 400), 0.0, 0), (599999, DEFAULT, 0.0, 0),
    (600001, DEFAULT, 0.0, 0), (1400003, DEFAULT, 0.0, 0), (1400003, (999, 99, 199, 201), 0.0, 0),
    (1400003, (4096, 3, 1, 33000), 0.0, 0)])
def test_sample_counts_what_the_separate_passes_count(n, cells, freq, thermal):
    from lokigpu import capi
    alone = _context(n, cells, freq, thermal)
    a = alone.solve()
    batched = _context(n, cells, freq, thermal)
    batch = capi.Batch(0, 1)
    batch.add(batched)
    res, status, _ = batch.run()
    assert status == [0]
    assert a.integration_points == res[0].integration_points and a.max_eedf_energy == res[0].max_eedf_energy
    d, e = alone.distributions(), batched.distributions()
    for k in ("eedf", "eadf", "evdf", "efadf", "esadf") + (("eedf_periodic",) if freq else ()):
        np.testing.assert_array_equal(d[k], e[k], err_msg=k)
    batch.close()
    alone.close()
    batched.close()


@pytest.mark.parametrize("n", [2, 31, 32, 65, 19455, 19457, 155647, 155649, 155681, 700001])
def test_every_electron_is_advanced_once_alone(n):
    """The solve alone spreads the ensemble over its warps by size (blocks of two
    warps, one electron per lane, shares and chunks of 32): collision counts equal
    the batched solve's, whose warps take chunks from a counter."""
    from lokigpu import capi
    alone = _context(n, DEFAULT, 0.0, 0)
    a = alone.solve()
    batched = _context(n, DEFAULT, 0.0, 0)
    batch = capi.Batch(0, 1)
    batch.add(batched)
    res, status, _ = batch.run()
    assert status == [0]
    assert (a.real_collisions, a.null_collisions) == (res[0].real_collisions, res[0].null_collisions)
    np.testing.assert_array_equal(alone.process_results()[0], batched.process_results()[0])
    batch.close()
    alone.close()
    batched.close()
