"""A context on its own with more electrons than its samples count the distributions of
(9e6: they are counted in passes of their own, between the intervals): every count
equals the batch's, which counts them with its samples, as in test_gpu_sample_dist."""
import numpy as np
import pytest

from test_gpu_sample_dist import DEFAULT, N_GAS, _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9000000, 9000001])
@pytest.mark.parametrize("freq", [0.0, N_GAS * 1e-14 / (2 * np.pi)])
def test_every_sample_is_counted_once(n, freq):
    from lokigpu import capi
    alone = _context(n, DEFAULT, freq, 0)
    a = alone.solve()
    batched = _context(n, DEFAULT, freq, 0)
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
