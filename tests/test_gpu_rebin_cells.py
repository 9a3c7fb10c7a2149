"""Every cell that the device's re-binning (k_rebin) leaves, against the reference's loop
over the old cells (BoltzmannMC.C:1495-1548) in numpy: the shares of an old cell that
reaches into two new ones, the per-phase sums that keep their old cells and take each
old cell once per phase. And a solve that re-bins.

Tolerances: EEDF and EADF add the same products in the same order, so only the rounding of
a share (1 ulp of two divisions and a difference of numbers up to the cell's index) may
differ: 1e-11 of the largest cell. The per-phase sums add a phase count times a sum where
the loop adds term by term, at most 64 x 4100 additions of 1.1e-16: 1e-10 of the
largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N_GAS = 3.22e22


def _loop(old_max, new_max, eedf, eadf, per):
    n = len(eedf)
    old, new = old_max / n, new_max / n
    e, a = np.zeros_like(eedf), np.zeros_like(eadf)
    p = per.copy()
    for o in range(n):
        lo = o * old
        hi = old_max if o + 1 == n else (o + 1) * old
        nl, nr = int(lo / new), int(hi / new)
        lf = 1.0 if nl == nr else (nr * new - lo) / old
        for cell, share in ((nl, lf),) + (((nr, 1.0 - lf),) if nl != nr else ()):
            e[cell] += share * eedf[o]
            a[cell] += share * eadf[o]
            for _ in range(per.shape[0]):
                p[:, cell] += share * per[:, o]
    return e, a, p


@pytest.fixture(scope="module")
def ctx():
    from lokigpu import capi
    c = capi.Context(capi.default_config(n_electrons=100.0, n_interp=100))
    yield c
    c.close()


@pytest.mark.parametrize("growth", [1.0 + 1e-9, 1.2, 1.37, 2.0, 2.9, 37.3])
@pytest.mark.parametrize("cells,cos,phases", [(1, 3, 2), (2, 1, 1), (37, 5, 3), (255, 100, 1), (257, 7, 64),
                                              (1000, 100, 16), (4096, 2, 2)])
def test_every_cell(ctx, cells, cos, phases, growth):
    rng = np.random.default_rng(cells + phases)
    eadf = rng.integers(0, 100000, (cells, cos)).astype(float)
    eedf = eadf.sum(axis=1) + rng.integers(0, 5, cells)
    per = rng.integers(0, 100000, (phases, cells)).astype(float)
    old_max = 23.7
    got = ctx.replay_rebin(old_max, growth * old_max, eedf, eadf, per)
    want = _loop(old_max, growth * old_max, eedf, eadf, per)
    for g, w, tol in zip(got, want, (1e-11, 1e-11, 1e-10)):
        assert np.max(np.abs(g - w)) <= tol * np.max(np.abs(w))
    assert abs(got[0].sum() - eedf.sum()) <= 1e-12 * eedf.sum()


def test_parts_alone(ctx):
    eedf = np.arange(1.0, 12.0)
    want = _loop(5.0, 6.5, eedf, np.zeros((11, 0)), np.zeros((0, 11)))[0]
    got, none, none_too = ctx.replay_rebin(5.0, 6.5, eedf)
    assert none is None and none_too is None and np.max(np.abs(got - want)) <= 1e-11 * want.max()


def test_refused(ctx):
    from lokigpu import capi
    for old, new, n in ((5.0, 5.0, 4), (5.0, 4.0, 4), (0.0, 1.0, 4), (1.0, float("nan"), 4), (1.0, 2.0, 4097)):
        with pytest.raises(capi.LokiGpuError):
            ctx.replay_rebin(old, new, np.ones(n))


def test_a_heating_swarm_re_bins():
    from lokigpu import capi, synth
    ps = synth.flatten([synth.atomic_gas()])
    grids = []
    for points in (1.0, 300.0):
        c = capi.Context(capi.default_config(n_electrons=400.0, n_interp=2000, seed=9, init_temp_ratio=1.0,
                                             max_coll_before_ss=1e-6, req_integration_points=points))
        c.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
        c.set_conditions(N_GAS, 300.0, 100.0)
        grids.append(c.solve().max_eedf_energy)
        c.close()
    assert grids[1] > grids[0] > 0  # the same trajectories, a wider grid after 300 samples
