"""Creating a batch or a server costs no more than creating a context of 10,000
electrons: one pinned and one device allocation, as large as their slots need.

Bound: 1.3 times the context's time (medians of 15 in turn): 0.85 and 1.0 measured, 1.45
and 1.6 with staging for the most slots and an allocation for each part."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_creation_costs_no_more_than_a_context():
    from lokigpu import capi

    def timed(make):
        t0 = time.perf_counter()
        h = make()
        (h.stop if hasattr(h, "stop") else h.close)()
        return time.perf_counter() - t0

    cfg = capi.default_config(n_electrons=10000.0, n_interp=10000)
    makes = [lambda: capi.Context(cfg), lambda: capi.Batch(0, 64), lambda: capi.Server(0, 16)]
    for m in makes:
        timed(m)
    t = np.median([[timed(m) for m in makes] for _ in range(15)], axis=0)
    assert t[1] <= 1.3 * t[0] and t[2] <= 1.3 * t[0], t * 1e6
