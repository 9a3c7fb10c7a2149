"""The sample of a context on its own about the ensemble from which its blocks keep EADF
and EVDF cells in shared memory (5250 electrons per SM): every count equals the batch's, as
in test_gpu_sample_dist."""
import numpy as np
import pytest

from test_gpu_sample_dist import DEFAULT, N_GAS, _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [-1, 0, 1])
@pytest.mark.parametrize("cells,freq", [(DEFAULT, 0.0), ((17, 100, 400, 400), N_GAS * 1e-14 / (2 * np.pi))])
def test_counts_about_the_edge(more, cells, freq):
    import torch
    from lokigpu import capi
    n = 5250 * torch.cuda.get_device_properties(0).multi_processor_count + more
    alone = _context(n, cells, freq, 0)
    a = alone.solve()
    batched = _context(n, cells, freq, 0)
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
