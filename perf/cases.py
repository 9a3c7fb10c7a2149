"""The work that a user of the electron Monte Carlo backend has it do, as timed cases.

Four kinds of call, all through the Python front end of the C ABI:

* ``solve``: one context (one gas mixture, one ensemble) solved for one E/N
  after the other, as a job list of the reference runs (``lgpu_solve``):
  thousands to millions of electrons, DC, crossed magnetic field and AC, cold
  and thermal targets.
* ``batch``: many swarm conditions in one ``lgpu_batch_run``: a sweep.
* ``served``: a handful of jobs of different random mixtures submitted to a
  running ``lgpu_server`` and waited for.
* ``post``: the EEDF post-processing of a solve's end (``lgpu_eedf_postprocess``)
  and of the per-phase EEDFs of an AC run (``lgpu_eedf_rates``).

Mixtures, fields, electron counts and numerics are the ones of bench.py and of
the tests. Every solve starts from a Maxwellian at kT = 1 eV and declares the
steady state at its first check (sample 128), then takes a given number of
integration points: the count of synchronisation intervals is known before.

What comes back: everything for gases without ionization and attachment, whose
trajectories are fixed by the seed. With them the order in which electrons are
replaced is not, so those cases solve several conditions and return each one's
swarm parameters and collisions per process, as averages (the rest is noise from
run to run, over so few samples: bulk coefficients, rates of hardly populated
states, distributions, whose grid follows the one fastest electron). The ensembles
are FP32 and so are the moments taken from them: those are handed on as FP32.
"""
import functools
import math
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "loki-mc_gb300", "python"))

from lokigpu import capi, synth  # noqa: E402

N_GAS = 3.22e22  # m^-3
T_GAS = 300.0    # K
KT_INIT = 1.0 / (8.617333262e-5 * T_GAS)  # initial temperature ratio of kT = 1 eV
FIRST_CHECK = 128  # the sample at which the steady state is first looked for
QE, ME = 1.6021766208e-19, 9.10938356e-31


# ------------------------------------------------------------------ mixtures
@functools.lru_cache(maxsize=None)
def gases(name):
    if name == "atomic":
        return [synth.atomic_gas()]
    if name == "reid":
        return [synth.reid_ramp_gas()]
    if name == "n2":
        return [synth.n2_like_gas(e_max=1e4)]
    # the sweep's mixture: 65 processes, ionization in both gases, attachment
    return [synth.n2_like_gas(fraction=0.8, e_max=1e4), synth.o2_like_gas(fraction=0.2, e_max=1e4)]


@functools.lru_cache(maxsize=None)
def processes(name):
    return synth.flatten(gases(name))


@functools.lru_cache(maxsize=64)
def random_mixture(seed):
    """1-5 random gases of 10-40 processes each (a served request's mixture)."""
    rng = np.random.default_rng(seed)
    ng = int(rng.integers(1, 6))
    fr = rng.dirichlet(np.ones(ng))
    return synth.flatten([synth.random_gas(10 * seed + g, f"R{g}", float(fr[g]), e_max=1e4) for g in range(ng)])


def replaces(name):
    """Whether the mixture ionizes or attaches (electrons are replaced)."""
    return name in ("n2", "mix")


def config(seed, electrons, case, phases=100):
    return capi.default_config(seed=int(seed), n_electrons=float(electrons), n_interp=10000, init_temp_ratio=KT_INIT,
                               n_phases=int(phases), gas_temperature_effect=int(case.get("thermal", 0)),
                               max_coll_before_ss=0.01, req_integration_points=float(case["integration"]))


def fields(lo, hi, n):
    return [lo] if n == 1 else [lo * (hi / lo) ** (k / (n - 1)) for k in range(n)]


def frequency(omega_n):
    return omega_n * N_GAS / (2.0 * math.pi)


# --------------------------------------------------------------------- cases
def listed():
    return [
        # the end of one DC solve of the molecular gas: its EEDF's rates and two-term parameters
        {"name": "post_n2", "kind": "post", "gas": "n2", "eedfs": 1, "cells": 1000, "max_ev": 60.0, "omega_n": 0.0,
         "mag_hx": 0.0},
        # the end of an AC solve of the mixture: the rates of every phase's EEDF
        {"name": "post_mix_phases", "kind": "post", "gas": "mix", "eedfs": 100, "cells": 1000, "max_ev": 80.0,
         "omega_n": 1e-14, "mag_hx": 0.0},
        # the reference's default ensemble size on its simplest gas: a quick look, bound by latency
        {"name": "solve_atomic_1e4", "kind": "solve", "gas": "atomic", "lo_td": 100.0, "hi_td": 100.0, "points": 1,
         "electrons": 10000, "angle": 180.0, "mag_hx": 0.0, "omega_n": 0.0, "thermal": 0, "phases": 100,
         "integration": 200},
        # a magnetised swarm of the mixture with thermal targets, an odd ensemble size
        {"name": "solve_mix_b_thermal", "kind": "solve", "gas": "mix", "lo_td": 80.0, "hi_td": 160.0, "points": 8,
         "electrons": 100003, "angle": 90.0, "mag_hx": 500.0, "omega_n": 0.0, "thermal": 1, "phases": 100,
         "integration": 200},
        # the ramp-model benchmark's low fields with smartActivation, few collisions per electron
        {"name": "solve_reid_smart", "kind": "solve", "gas": "reid", "lo_td": 12.0, "hi_td": 24.0, "points": 2,
         "electrons": 33333, "angle": 180.0, "mag_hx": 0.0, "omega_n": 0.0, "thermal": 2, "phases": 100,
         "integration": 200},
        # the largest single ensembles of the request stream
        {"name": "solve_atomic_4e6", "kind": "solve", "gas": "atomic", "lo_td": 100.0, "hi_td": 100.0, "points": 1,
         "electrons": 4000000, "angle": 180.0, "mag_hx": 0.0, "omega_n": 0.0, "thermal": 0, "phases": 100,
         "integration": 200},
        # the single-condition benchmark's ensemble over a short E/N list, one solve after the other
        {"name": "solve_n2_1e6", "kind": "solve", "gas": "n2", "lo_td": 120.0, "hi_td": 240.0, "points": 8,
         "electrons": 1000000, "angle": 180.0, "mag_hx": 0.0, "omega_n": 0.0, "thermal": 0, "phases": 100,
         "integration": 200},
        # a phase-resolved AC run
        {"name": "solve_atomic_ac", "kind": "solve", "gas": "atomic", "lo_td": 100.0, "hi_td": 150.0, "points": 2,
         "electrons": 200000, "angle": 180.0, "mag_hx": 0.0, "omega_n": 1e-14, "thermal": 0, "phases": 64,
         "integration": 200},
        # many small conditions: a map of the molecular gas
        {"name": "batch_small", "kind": "batch", "gas": "n2", "conditions": 32, "lo_td": 20.0, "hi_td": 200.0,
         "lo_n": 10000, "hi_n": 30000, "branches": "dc", "thermal": 0, "integration": 200},
        # crossed magnetic field and AC side by side, equal ensembles
        {"name": "batch_field", "kind": "batch", "gas": "mix", "conditions": 32, "lo_td": 100.0, "hi_td": 150.0,
         "lo_n": 500000, "hi_n": 500000, "branches": "b+ac", "thermal": 0, "integration": 200},
        # the headline sweep: 64 points over 1..1000 Td, uneven ensembles
        {"name": "batch_sweep", "kind": "batch", "gas": "mix", "conditions": 64, "lo_td": 1.0, "hi_td": 1000.0,
         "lo_n": 10000, "hi_n": 2000000, "branches": "dc", "thermal": 0, "integration": 200},
        # jobs of unrelated mixtures that arrive together
        {"name": "served_mixtures", "kind": "served", "jobs": 16, "mixture": 2024, "lo_td": 10.0, "hi_td": 500.0,
         "lo_n": 20000, "hi_n": 500000, "integration": 200},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "post", "post", "batch", "batch", "served"])
    if kind == "post":
        gas = rng.choice(["atomic", "n2", "mix"])
        return {"kind": "post", "gas": gas, "eedfs": int(_log(rng, 1, 100)), "cells": int(_log(rng, 100, 2000)),
                "max_ev": _log(rng, 20.0, 200.0), "omega_n": rng.choice([0.0, _log(rng, 1e-16, 1e-14)]),
                "mag_hx": rng.choice([0.0, rng.uniform(100.0, 2000.0)])}
    if kind == "solve":
        gas = rng.choice(["atomic", "atomic", "reid", "n2", "mix"])
        lo = {"atomic": 40.0, "reid": 6.0, "n2": 40.0, "mix": 40.0}[gas] * rng.uniform(1.0, 2.5)
        branch = rng.choice(["dc", "dc", "b"] if replaces(gas) else ["dc", "dc", "b", "ac"])
        points = rng.randrange(6, 9) if replaces(gas) else rng.randrange(1, 4)
        top = 1000000 if replaces(gas) else 4000000 // points
        return {"kind": "solve", "gas": gas, "lo_td": lo, "hi_td": lo * rng.uniform(1.2, 2.0), "points": points,
                "electrons": int(_log(rng, 50000 if replaces(gas) else 8000, top)), "angle": 90.0 if branch == "b" else 180.0,
                "mag_hx": rng.uniform(100.0, 2000.0) if branch == "b" else 0.0,
                "omega_n": 1e-14 if branch == "ac" else 0.0, "thermal": rng.choice([0, 0, 1, 2]),
                "phases": rng.choice([16, 64]) if branch == "ac" else 100, "integration": rng.randrange(100, 201)}
    if kind == "batch":
        n = rng.randrange(12, 65)
        hi = int(_log(rng, 30000, 19000000 / n))
        lo_td = _log(rng, 20.0, 100.0)
        return {"kind": "batch", "gas": rng.choice(["n2", "mix"]), "conditions": n, "lo_td": lo_td,
                "hi_td": lo_td * rng.uniform(1.5, 6.0), "lo_n": max(15000, int(hi * rng.uniform(0.3, 1.0))), "hi_n": hi,
                "branches": rng.choice(["dc", "dc", "b+ac"]), "thermal": rng.choice([0, 0, 0, 2]),
                "integration": rng.randrange(120, 201)}
    return {"kind": "served", "jobs": rng.randrange(8, 25), "mixture": rng.randrange(1, 1000000),
            "lo_td": 10.0, "hi_td": _log(rng, 100.0, 500.0), "lo_n": int(_log(rng, 20000, 50000)),
            "hi_n": int(_log(rng, 60000, 500000)), "integration": rng.randrange(120, 201)}


# ---------------------------------------------------------------- conditions
def sizes(case, n):
    """Electron counts of a batch's or stream's conditions, log-uniform."""
    rng = np.random.default_rng(2024)
    lo, hi = math.log10(case["lo_n"]), math.log10(case["hi_n"])
    return [int(round(v)) for v in 10.0 ** rng.uniform(lo, hi, n)]


def batch_conditions(case):
    """(gas, E/N in Td, electrons, angle, frequency in Hz, B/N in Hx). The AC
    conditions take the atomic gas: their window ends within a period, where a
    step of the interval that follows the fastest electron would show."""
    n, gas = case["conditions"], case["gas"]
    td, ne = fields(case["lo_td"], case["hi_td"], n), sizes(case, n)
    if case["branches"] == "dc":
        return [(gas, td[k], ne[k], 180.0, 0.0, 0.0) for k in range(n)]
    nb = n // 2
    b = [(gas, case["lo_td"], ne[k], 90.0, 0.0, 2000.0 * k / max(nb - 1, 1)) for k in range(nb)]
    w = np.logspace(-15.0, -14.0, n - nb)
    return b + [("atomic", case["hi_td"], ne[nb + k], 180.0, frequency(float(w[k])), 0.0) for k in range(n - nb)]


def twoterm(name):
    """The collision behind each process, as the EEDF post-processing reads it."""
    out = []
    for g in gases(name):
        for c in g.collisions:
            e, v = np.asarray(c.energies, float), np.asarray(c.values, float)
            if c.ctype == "Elastic" and e[0] != 0:
                e, v = np.concatenate([[0.0], e]), np.concatenate([[v[0]], v])
            q = dict(kind=0 if c.ctype == "Elastic" else 1, ion={"Ionization": 1, "Attachment": 2}.get(c.ctype, 0),
                     density=g.density(c.target), threshold=c.threshold, mass_ratio=ME / g.mass,
                     stat_ratio=g.states[c.target].weight / g.states[c.product].weight if c.reverse else 0.0,
                     int_e=e, int_v=v, mom_e=e, mom_v=v / (1.0 + 0.02 * e))
            out.append(q)
            if c.reverse:
                out.append(dict(q, kind=2, density=g.density(c.product)))
    return out


def post_eedfs(case, seed):
    """Smooth EEDFs (eV^-3/2) as a solve leaves them: a spread of temperatures
    with a depleted tail, normalised on the cells."""
    rng = np.random.default_rng(seed)
    n, nc, top = case["eedfs"], case["cells"], case["max_ev"]
    step = top / nc
    e = (np.arange(nc) + 0.5) * step
    t = top * rng.uniform(0.04, 0.1, (n, 1))
    f = np.exp(-e / t - (e / (4.0 * t)) ** 2) * (1.0 + 0.1 * rng.uniform(-1.0, 1.0, (n, nc)))
    return f / (np.sum(f * np.sqrt(e), axis=1, keepdims=True) * step)


# ------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "post":
        ctx = capi.Context(capi.default_config(n_electrons=1000.0, n_interp=1000, n_energy_cells=case["cells"]))
        ps = processes(case["gas"])
        ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
        ctx.set_conditions(N_GAS, T_GAS, 100.0, 180.0, frequency(case["omega_n"]), case["mag_hx"])
        ctx.set_twoterm(twoterm(case["gas"]))
        return {"case": case, "ctx": ctx, "eedf": post_eedfs(case, seed)}
    if kind == "solve":
        ps = processes(case["gas"])
        ctx = capi.Context(config(seed, case["electrons"], case, case["phases"]))
        ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
        return {"case": case, "ctx": ctx}
    if kind == "batch":
        ctxs = []
        for k, (gas, td, ne, angle, freq, mag) in enumerate(batch_conditions(case)):
            ps = processes(gas)
            ctx = capi.Context(config(seed * 1000 + k, ne, case, 64))
            ctx.set_processes(ps, ps.gas_first, ps.gas_last, ps.gas_fraction)
            ctx.set_conditions(N_GAS, T_GAS, td, angle, freq, mag)
            ctxs.append(ctx)
        return {"case": case, "ctxs": ctxs, "batch": capi.Batch(0, len(ctxs))}
    ne = sizes(case, case["jobs"])
    td = fields(case["lo_td"], case["hi_td"], case["jobs"])
    jobs = [(config(seed * 1000 + k, ne[k], case, 16), random_mixture(case["mixture"] % 100000 + k), td[k])
            for k in range(case["jobs"])]
    return {"case": case, "jobs": jobs, "server": capi.Server(0, case["jobs"], 40e9)}


def swarm(results):
    f32 = np.float32
    return {"mean_energy": np.array([r.mean_energy for r in results], f32),
            "flux_velocity": np.array([r.flux_v[:] for r in results], f32),
            "flux_diffusion": np.array([r.flux_d[:] for r in results], f32)}


def frequencies(results, counts, electrons):
    """Collisions per process, electron and second (s^-1) since the steady state."""
    return [c / (float(n) * (r.final_time - r.ss_time)) for r, c, n in zip(results, counts, electrons)]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "post":
        ctx, f = state["ctx"], state["eedf"]
        if len(f) > 1:
            return {"rates": ctx.eedf_rates(f, case["max_ev"])}
        params, rates = ctx.eedf_postprocess(f[0], case["max_ev"])
        return {"rates": rates, "params": params.values()}
    if kind == "solve":
        ctx, results, procs, dists = state["ctx"], [], [], []
        for td in fields(case["lo_td"], case["hi_td"], case["points"]):
            ctx.set_conditions(N_GAS, T_GAS, td, case["angle"], frequency(case["omega_n"]), case["mag_hx"])
            results.append(ctx.solve())
            procs.append(ctx.process_results())
            dists.append(ctx.distributions())
        out = swarm(results)
        if replaces(case["gas"]):
            out["collisions"] = np.array(frequencies(results, [p[0] for p in procs], [case["electrons"]] * len(procs)))
        else:
            out["rates"] = np.array([p[1] for p in procs])
            out["counts"] = np.array([p[0] for p in procs]).astype(np.int64)
            out["power"] = np.array([np.concatenate([[r.power_field], p[2], p[3]]) for r, p in zip(results, procs)],
                                    np.float32)
            for k in ("eedf", "eadf", "evdf"):
                out[k] = np.array([d[k] for d in dists])
        return out
    if kind == "batch":
        batch, ctxs = state["batch"], state["ctxs"]
        for ctx in ctxs:
            batch.add(ctx)
        results, status, _ = batch.run()
        if any(status):
            raise RuntimeError(f"a condition failed: {status}")
        out = swarm(results)
        counts = [ctx.process_results()[0] for ctx in ctxs]
        out["collisions"] = np.concatenate(frequencies(results, counts, sizes(case, len(ctxs))))
        return out
    srv = state["server"]
    ids = [srv.submit(cfg, ps, ps.gas_first, ps.gas_last, ps.gas_fraction, N_GAS, T_GAS, td)
           for cfg, ps, td in state["jobs"]]
    done = [srv.wait(i, 60.0) for i in ids]
    if any(s.state != capi.JOB_DONE for s in done):
        raise RuntimeError("a job failed: " + "; ".join(s.error.decode(errors="replace") for s in done))
    out = swarm([s.result for s in done])
    counts = [srv.rates(i, ps.n)[0] for i, (_, ps, _) in zip(ids, state["jobs"])]
    out["collisions"] = np.concatenate(frequencies([s.result for s in done], counts, sizes(case, len(done))))
    return out


# ----------------------------------------------------------------------- work
def work(case):
    """A solve reads and writes each electron's 32-byte state once per
    synchronisation interval (position, velocity, remaining flight) and makes
    about one trial event and two flights in it: some 35 operations. The
    post-processing reads the EEDFs and cross sections once and sums every process
    over every cell."""
    if case["kind"] == "post":
        tabs = sum(len(q["int_e"]) for q in twoterm(case["gas"]))
        p, nc, n = processes(case["gas"]).n, case["cells"], case["eedfs"]
        return {"bytes": 8.0 * (4 * tabs + n * nc + n * p + 16), "flops": 20.0 * p * nc + 4.0 * p * nc * n}
    if case["kind"] == "solve":
        total = case["electrons"] * case["points"]
    else:
        total = sum(sizes(case, case["conditions"] if case["kind"] == "batch" else case["jobs"]))
    steps = float(total) * (FIRST_CHECK - 2 + case["integration"])
    return {"bytes": 64.0 * steps, "flops": 35.0 * steps}


# ---------------------------------------------------------------------- exact
def _interp(e, v, x):
    """Linear between the raw points, zero outside the table."""
    return np.where((x < e[0]) | (x > e[-1]), 0.0, np.interp(x, e, v))


def exact(case, seed):
    """The post-processing in 64 bits; a Monte Carlo run has no exact value."""
    if case["kind"] != "post":
        return None
    nc, top = case["cells"], case["max_ev"]
    eedfs = post_eedfs(case, seed)
    step = top / nc
    node = np.arange(nc + 1) * step
    node[-1] = top
    cell = np.linspace(0.5 * step, top - 0.5 * step, nc)
    speed = math.sqrt(2.0 * QE / ME)
    procs = twoterm(case["gas"])
    rates = np.zeros((len(eedfs), len(procs)))
    mt, er, erc = np.zeros(nc + 1), np.zeros(nc + 1), np.zeros(nc + 1)
    sig = None
    with np.errstate(divide="ignore", invalid="ignore"):
        inv = np.where(node > 0, 1.0 / node, 0.0)
    for p, q in enumerate(procs):
        thr, first = q["threshold"], int(math.floor(q["threshold"] / step))
        if q["kind"] == 2:
            up = (1.0 + thr * inv) * q["stat_ratio"] * q["density"] * (node > 0)
            s_int, s_mom = _interp(q["int_e"], q["int_v"], node + thr) * up, _interp(q["mom_e"], q["mom_v"], node + thr) * up
            mt, er, erc = mt + s_mom, er + s_int * thr * inv, erc + s_int
            w = 0.5 * (sig[first:-1] + sig[first + 1:]) * cell[first:]
            rates[:, p] = speed * q["stat_ratio"] * step * (eedfs[:, :nc - first] @ w)
            continue
        on = np.ones(nc + 1, bool) if q["kind"] == 0 else node > thr
        sig = np.where(on, _interp(q["int_e"], q["int_v"], node), 0.0)
        mt = mt + np.where(on, _interp(q["mom_e"], q["mom_v"], node), 0.0) * q["density"]
        if q["kind"] == 0:
            er = er + 2.0 * q["mass_ratio"] * sig * q["density"]
        else:
            er, erc = er + sig * q["density"] * thr * inv, erc + sig * q["density"]
        w = 0.5 * (sig[first:-1] + sig[first + 1:]) * cell[first:]
        rates[:, p] = speed * step * (eedfs[:, first:] @ w)
    if len(eedfs) > 1:
        return {"rates": rates}
    k = [sum(q["density"] * rates[0, p] for p, q in enumerate(procs) if q["kind"] != 2 and q["ion"] == i) for i in (1, 2)]
    f, third = eedfs[0], speed / 3.0
    wl, wc = 2.0 * math.pi * frequency(case["omega_n"]), QE * case["mag_hx"] * 1e-27 * N_GAS / ME
    pre = N_GAS * speed * step
    mid = [np.sum(f * cell * 0.5 * (a[1:] + a[:-1])) * pre for a in (mt, er, erc)]
    mta = mt.copy()
    mta[1:] += (k[0] - k[1]) / (speed * np.sqrt(node[1:]))
    u, m, df = node[1:nc], mta[1:nc], f[1:] - f[:-1]
    de, d = (2.0 * third * step * np.sum(cell ** n * f / (mta[:-1] + mta[1:])) for n in (2, 1))
    me, mo = (-third * np.sum(u ** n * df / m) for n in (2, 1))
    a = -2.0 / 3.0 * QE / ME * u ** 1.5 * df
    nu = N_GAS * m * speed * np.sqrt(u)
    both = (nu ** 2 + (wl - wc) ** 2) * (nu ** 2 + (wl + wc) ** 2)
    params = [k[0], k[1], *mid, de, me, d, mo, d / mo,
              N_GAS * np.sum(nu * (nu ** 2 + wl ** 2 + wc ** 2) / both * a),
              -N_GAS * np.sum(wl * (nu ** 2 + wl ** 2 - wc ** 2) / both * a),
              -N_GAS * wc * np.sum((nu ** 2 - wl ** 2 + wc ** 2) / both * a),
              N_GAS * 2.0 * wl * wc * np.sum(nu / both * a),
              N_GAS * np.sum(nu / (nu ** 2 + wl ** 2) * a), -N_GAS * np.sum(wl / (nu ** 2 + wl ** 2) * a)]
    return {"rates": rates[0], "params": np.array(params)}
