"""The tables built on the device about the sizes where its blocks change their number
of warps (as many blocks of 32 rows as SMs; so many processes that one block fills an
SM's shared memory), against the oracle as in test_gpu_table_edges."""
import os
import sys

import numpy as np
import pytest

import golden_util as gu
from test_gpu_table_edges import DENSITY, _arrays

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,P", [("atomic", 1), ("mix", 0), ("n2", 293), ("n2", 294)])
@pytest.mark.parametrize("more", [0, 1, 33])
def test_tables_about_the_edges(case, P, more):
    import oracle as O
    import torch
    from lokigpu import capi
    M = 32 * torch.cuda.get_device_properties(0).multi_processor_count + more
    a = _arrays(case, P)
    ps = gu.processes(a)
    ctx = capi.Context(capi.default_config(n_electrons=100.0, n_interp=M))
    ctx.set_processes(ps, a["gas_first"], a["gas_last"], a["gas_frac"])
    ctx.set_conditions(DENSITY, 300.0, 100.0)
    nu_tot, nu_max, sig, cum = ctx.build_tables(97.0, M, ps.n)
    pr = O.OracleProcs(a, M)
    pr.build_tables(O.make_fields(DENSITY, 300.0), 97.0)
    assert np.array_equal(sig, pr.sig.astype(np.float32))
    assert np.array_equal(cum, pr.cum.astype(np.float32))
    np.testing.assert_allclose(nu_tot, pr.nu_tot, rtol=1e-15, atol=0)
    np.testing.assert_array_equal(nu_max, np.maximum.accumulate(nu_tot))
    ctx.close()
