"""Population control (BoltzmannMC.C:1282-1408) where one kind of event outnumbers
the other: a gas that mostly attaches (slots clone other electrons), one that mostly
ionizes (electrons are removed at random), one where both nearly balance, alone and
in a batch, with and without spilled secondaries, against the CPU oracle's runs.

Compared: the mean energy within five combined standard errors plus 1 % (the
device places secondaries at the synchronisation time), each rate coefficient within
five combined Poisson errors doubled for autocorrelation plus 2 %: the bounds that
the batch tests use, widened by one standard error for the oracle's smaller run."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))

pytestmark = pytest.mark.gpu
N_GAS = 3.22e22
KT = 1.0 / (8.617333262e-5 * 300.0)


def _processes(att, ion):
    from lokigpu import synth
    e = synth.log_grid(100)
    gas = synth.atomic_gas()
    gas.collisions = [synth.Collision("Elastic", "A1(gnd)", "A1(gnd)", 0.0, e, np.full_like(e, 5e-20)),
                      synth.Collision("Attachment", "A1(gnd)", "A1(-)", 1.0, e, np.where(e < 1.0, 0.0, att)),
                      synth.Collision("Ionization", "A1(gnd)", "A1(+)", 12.0, e, np.where(e < 12.0, 0.0, ion))]
    gas.states = {"A1(gnd)": synth.State(1.0), "A1(-)": synth.State(0.0), "A1(+)": synth.State(0.0)}
    return synth.flatten([gas])


def _oracle(ps, n):
    import oracle as O
    off = np.concatenate([[0], np.cumsum([len(x) for x in ps.raw_e])]).astype(np.int32)
    arrays = dict(ptype=ps.ptype, is_super=ps.is_super, sampler=ps.sampler, sampler_p0=ps.sampler_p0,
                  sampler_p1=ps.sampler_p1, superw=ps.superw, emin=ps.emin, emax=ps.emax, rel_dens=ps.rel_dens,
                  mass=ps.mass, red_mass=ps.red_mass, eloss=ps.eloss, wparam=ps.wparam, raw_off=off[:-1],
                  raw_len=np.array([len(x) for x in ps.raw_e], np.int32), raw_e=np.concatenate(ps.raw_e),
                  raw_v=np.concatenate(ps.raw_v), gas_first=ps.gas_first, gas_last=ps.gas_last,
                  gas_frac=ps.gas_fraction, energy_max_elastic=ps.energy_max_elastic)
    pr = O.OracleProcs(arrays, 2000)
    f = O.make_fields(N_GAS, 300.0, E=(0.0, 0.0, -200.0 * 1e-21 * N_GAS))
    cfg = O.default_run_config(n, n_threads=4, seed=5, req_integration_points=600.0, init_temp_ratio=KT,
                               max_coll_before_ss=40.0)
    st, res, out = O.run(pr, f, cfg)
    assert st == 0
    return res, out["rate"]


@pytest.mark.parametrize("att,ion", [(2e-21, 1e-22), (1e-22, 4e-20), (1e-21, 2e-20)])
def test_population_control_against_the_oracle(att, ion):
    from lokigpu import capi
    ps = _processes(att, ion)
    ref, ref_rate = _oracle(ps, 10000)
    runs = []
    for how in ("alone", "spill", "batch", "batch spill"):
        cfg = capi.default_config(n_electrons=30011.0, n_interp=2000, seed=6, init_temp_ratio=KT,
                                  req_integration_points=600.0, max_coll_before_ss=40.0,
                                  advance_queue=1 if "spill" in how else 0)
        ctx = capi.Context(cfg)
        ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
        ctx.set_conditions(N_GAS, 300.0, 200.0)
        if "batch" in how:
            batch = capi.Batch(0, 1)
            batch.add(ctx)
            res, status, _ = batch.run()
            assert status == [0], ctx.last_error()
            r = res[0]
            batch.close()
        else:
            r = ctx.solve()
        runs.append((how, r, ctx.process_results()))
        ctx.close()
    for how, r, (counts, rate, _, _) in runs:
        err = np.hypot(r.mean_energy_err, ref.mean_energy_err)
        assert abs(r.mean_energy - ref.mean_energy) <= 5.0 * err + 0.01 * ref.mean_energy, (how, r.mean_energy, ref.mean_energy)
        for p in range(len(rate)):
            if counts[p] < 2000:
                continue
            ref_counts = counts[p] * 10000.0 / 30011.0
            rel = 2.0 * 5.0 * np.sqrt(1.0 / counts[p] + 1.0 / ref_counts) + 0.02
            assert abs(rate[p] - ref_rate[p]) <= rel * ref_rate[p], (how, p, rate[p], ref_rate[p], rel)
