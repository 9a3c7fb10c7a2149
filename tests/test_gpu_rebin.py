"""The re-binning of the energy tallies when an electron outgrows the grid
(BoltzmannMC.C:1495-1548): small ensembles re-bin often. Every old cell's count goes to
the new cells in full, so the EADF's rows keep summing to the EEDF and the EEDF to
one; no count strays further than the width of a last cell, so the mean energy over the
grid stays the sampled one within a cell; the per-phase EEDFs, which keep their old
cells and take each once per phase (:1523-1541), stay normalised.

Tolerances: sums of up to 4096 x 100 terms in FP64, 1e-11; the mean energy within one
cell's width plus the spread of the shares (two widths)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N_GAS = 3.22e22


@pytest.mark.parametrize("n,cells,cos,phases", [(50, 1000, 100, 0), (400, 4096, 100, 0), (400, 1, 7, 0), (400, 37, 3, 1),
                                                (3000, 1000, 100, 16)])
def test_counts_are_kept(n, cells, cos, phases):
    from lokigpu import capi, synth
    ps = synth.flatten([synth.atomic_gas()])
    cfg = capi.default_config(n_electrons=float(n), n_interp=2000, seed=9, init_temp_ratio=1.0, n_energy_cells=cells,
                              n_cos_cells=cos, n_phases=max(phases, 1), max_coll_before_ss=1e-6,
                              req_integration_points=300.0)
    ctx = capi.Context(cfg)
    ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
    ctx.set_conditions(N_GAS, 300.0, 100.0, 180.0, N_GAS * 1e-14 / (2 * np.pi) if phases else 0.0, 0.0)
    r = ctx.solve()
    d = ctx.distributions()
    e, f = d["eedf_cells"], d["eedf"]
    width = r.max_eedf_energy / cells
    # the swarm heats from 300 K after the grid was set: the grid grew
    series = ctx.series(1, 1)[r.first_integration_index:]
    assert abs(np.sum(f * np.sqrt(e)) * width - 1.0) <= 1e-11
    rows = np.sum(d["eadf"], axis=1) * (2.0 / cos) / 2.0
    assert np.all(np.abs(rows - f) <= 1e-11 * np.abs(f).max())
    mean = np.sum(f * e * np.sqrt(e)) * width
    assert abs(mean - series.mean()) <= 3.0 * width, (mean, series.mean(), width)
    if phases:
        per = d["eedf_periodic"]
        seen = np.isfinite(per).all(axis=1)
        assert seen.any()
        assert np.all(per[seen] >= 0)
        assert np.allclose(np.sum(per[seen] * np.sqrt(e), axis=1) * width, 1.0, rtol=0, atol=1e-11)
    ctx.close()
