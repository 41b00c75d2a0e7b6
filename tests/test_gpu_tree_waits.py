"""Grid barriers of the device tree that run out, with no fault (the test hook
makes its first CTA leave before the first barrier): reported as PGF_ERR_DEVICE
at once, and the handle works again afterwards."""
from __future__ import annotations

import time

import numpy as np
import pytest

from petar_gb300 import gpuforce, ics, nbody

pytestmark = pytest.mark.gpu

LIMIT_NS = 2_000_000


class _stalled:
    def __enter__(self):
        gpuforce.set_wait_limit_ns(LIMIT_NS)
        gpuforce.test_stall_producer(1)

    def __exit__(self, *exc):
        gpuforce.test_stall_producer(0)
        gpuforce.set_wait_limit_ns(0)


@pytest.mark.parametrize("graph", [None, False, True])
def test_tree_barrier_that_runs_out_is_a_device_error(graph):
    cl = ics.make_king_cluster(4, 3000, 0.01, W0=6.0, theta=0.5)
    with nbody.DeviceNBody(cl) as h:
        before = h.state()
        if graph:
            h.run(1, 0.0)  # captures the step; the limit below must reach it all the same
        with _stalled():
            t0 = time.perf_counter()
            with pytest.raises(gpuforce.GpuForceError) as e:
                h.force() if graph is None else h.run(1, 0.0, graph=graph)
            assert e.value.code == 6, e.value  # PGF_ERR_DEVICE
            assert "room" not in str(e.value)
            assert time.perf_counter() - t0 < 1.0  # one attempt: a rebuild would wait again
        h.force()
        after = h.state()
        for k in ("acc", "pot", "n_ngb"):
            np.testing.assert_array_equal(after[k], before[k], err_msg=k)


def test_tree_barrier_that_runs_out_fails_creation():
    cl = ics.make_king_cluster(4, 3000, 0.01, W0=6.0, theta=0.5)
    with _stalled():
        t0 = time.perf_counter()
        with pytest.raises(gpuforce.GpuForceError) as e:
            nbody.DeviceNBody(cl)
        assert e.value.code == 6, e.value
        assert time.perf_counter() - t0 < 1.0
