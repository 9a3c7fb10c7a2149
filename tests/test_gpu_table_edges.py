"""The tables built on the device at the sizes where their blocks' work changes hands
(32 rows per block, a run of rows per warp of the running maximum, 256 null-test
bounds; one process to the most a context takes), against the oracle's: sums in
process order, every step rounded as the reference's, so the FP32 values are equal
and the FP64 ones differ by the rounding of a square root at most."""
import os
import sys

import numpy as np
import pytest

import golden_util as gu

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))

pytestmark = pytest.mark.gpu
DENSITY = 3.22e22


def _arrays(case, P):
    """A golden case's processes; P > 0: its elastic one, then one inelastic process
    again and again with a growing threshold, P in all."""
    a = gu.proc_arrays(gu.load(case))
    if not P:
        return a
    el = int(np.nonzero(a["is_elastic"])[0][0])
    inel = [p for p in range(len(a["ptype"])) if not a["is_elastic"][p] and not a["is_super"][p] and a["ptype"][p] == 0][0]
    pick = np.array([el] + [inel] * (P - 1))
    n = len(a["ptype"])
    out = {k: (v[pick] if isinstance(v, np.ndarray) and v.ndim == 1 and len(v) == n else v) for k, v in a.items()}
    out["gas_first"], out["gas_last"], out["gas_frac"] = np.array([0]), np.array([P - 1]), np.array([1.0])
    out["emin"] = out["emin"] + 0.01 * np.arange(P) * (np.arange(P) > 0)
    return out


@pytest.mark.parametrize("case,P,M", [("mix", 0, m) for m in (2, 31, 32, 33, 255, 257, 1024, 1025, 4097)] +
                         [("atomic", 1, 1000), ("atomic", 2, 1000), ("n2", 63, 321), ("n2", 64, 321), ("n2", 511, 97),
                          ("n2", 512, 97)])
def test_tables_against_the_oracle(case, P, M):
    import oracle as O
    from lokigpu import capi
    a = _arrays(case, P)
    ps = gu.processes(a)
    ctx = capi.Context(capi.default_config(n_electrons=100.0, n_interp=M))
    ctx.set_processes(ps, a["gas_first"], a["gas_last"], a["gas_frac"])
    ctx.set_conditions(DENSITY, 300.0, 100.0)
    for top in (37.0, 411.0):
        nu_tot, nu_max, sig, cum = ctx.build_tables(top, M, ps.n)
        pr = O.OracleProcs(a, M)
        pr.build_tables(O.make_fields(DENSITY, 300.0), top)
        assert np.array_equal(sig, pr.sig.astype(np.float32))
        assert np.array_equal(cum, pr.cum.astype(np.float32))
        np.testing.assert_allclose(nu_tot, pr.nu_tot, rtol=1e-15, atol=0)
        np.testing.assert_array_equal(nu_max, np.maximum.accumulate(nu_tot))
    ctx.close()
