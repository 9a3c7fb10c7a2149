"""The device's EEDF post-processing at the sizes where its blocks' work changes
hands: cell counts around a tile of cells and a block of the parameter sums,
EEDF counts around the warps of a block and the EEDFs of a block, raw tables
that are staged in shared memory and ones that are not; against the oracle's
FP64 post-processing.

Tolerance: every summed term has the same sign (a falling EEDF, no field
frequency), so a sum of n terms in another order differs by at most n x 2^-53
relative on each side, 4.6e-13 for both at 2049 cells, plus a few roundings."""
import os
import sys

import numpy as np
import pytest

import golden_util as gu

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
import eedf_post as E  # noqa: E402

pytestmark = pytest.mark.gpu
REL = 1e-12
DENSITY = 3.22e22


def _case(points):
    """A context of the N2-like golden gas and its two-term inputs, the raw tables
    resampled on `points` energies (0: as they are)."""
    from lokigpu import capi
    d = dict(np.load(os.path.join(HERE, "golden", "eedf_post_n2_dc200.npz")))
    procs = E.procs_from_fixture(d)
    if points:
        for q in procs:
            for e, v in (("int_e", "int_v"), ("mom_e", "mom_v")):
                grid = np.linspace(q[e][0], q[e][-1], points)
                q[e], q[v] = grid, np.interp(grid, q[e], q[v])
    arrays = {k[5:]: v for k, v in d.items() if k.startswith("proc_")}
    arrays["energy_max_elastic"] = 1e3
    ctx = capi.Context(capi.default_config(n_electrons=1000.0, n_interp=1000))
    ctx.set_processes(gu.processes(arrays), arrays["gas_first"], arrays["gas_last"], arrays["gas_frac"])
    ctx.set_conditions(DENSITY, 300.0, 100.0)
    ctx.set_twoterm(procs)
    return ctx, procs


def _eedfs(n, cells, top):
    e = (np.arange(cells) + 0.5) * top / cells
    t = np.linspace(2.0, 6.0, n)[:, None]
    f = np.exp(-e / t)
    return f / (np.sum(f * np.sqrt(e), axis=1, keepdims=True) * top / cells)


@pytest.mark.parametrize("points", [0, 512, 513])
@pytest.mark.parametrize("cells", [2, 31, 33, 512, 1024, 1025, 2049])
def test_one_eedf(cells, points):
    ctx, procs = _case(points)
    f = _eedfs(1, cells, 50.0)[0]
    for _ in range(2):  # the second call finds the ticket as the first left it
        out, rates = ctx.eedf_postprocess(f, 50.0)
        ref_rates, ref, _ = E.postprocess(f, 50.0, 0.0, 0.0, DENSITY, procs)
        assert np.all(np.abs(rates - ref_rates) <= REL * np.abs(ref_rates))
        assert np.all(np.abs(out.values() - ref) <= REL * np.abs(ref)), (out.values(), ref)
    ctx.close()


@pytest.mark.parametrize("n", [2, 3, 8, 9, 16, 17, 300, 2100])
def test_many_eedfs(n):
    ctx, procs = _case(0)
    cells = 1025 if n < 20 else 37
    f = _eedfs(n, cells, 40.0)
    rates = ctx.eedf_rates(f, 40.0)
    for k in sorted({0, n // 2, n - 2, n - 1}):
        ref = E.postprocess(f[k], 40.0, 0.0, 0.0, DENSITY, procs)[0]
        assert np.all(np.abs(rates[k] - ref) <= REL * np.abs(ref)), k
    ctx.close()
