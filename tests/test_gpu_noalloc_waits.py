"""A bounded wait of the pair kernel that runs out, with no fault (the same
test hook as the dispatch path's: producers stop after a number of items): the
allocation-free call, which has returned by then and has no status to report it
in, still leaves complete results."""
from __future__ import annotations

import pytest

import oracle
from helpers import assert_mixed_parity
from petar_gb300 import gpuforce, ics, walks
from test_zz_no_alloc import _call, _device_inputs, _lib

pytestmark = pytest.mark.gpu

LIMIT_NS = 2_000_000


class _stalled:
    def __enter__(self):
        gpuforce.set_wait_limit_ns(LIMIT_NS)
        gpuforce.test_stall_producer(1)

    def __exit__(self, *exc):
        gpuforce.test_stall_producer(0)
        gpuforce.set_wait_limit_ns(0)


@pytest.mark.parametrize("n", [700, 8192])
def test_noalloc_completes_when_a_wait_runs_out(n):
    torch = pytest.importorskip("torch")
    wb = walks.build_walks(ics.make_plummer_cluster(3, n, 0.02, binary_fraction=0.3))
    o = oracle.force(wb)
    f, d = _lib(), _device_inputs(torch, wb)
    for stalled in (True, True, False):
        if stalled:
            with _stalled():
                rc, msg, accp, nnb = _call(f, torch, wb, d)
        else:
            rc, msg, accp, nnb = _call(f, torch, wb, d)
        assert rc == 0, msg
        assert_mixed_parity(accp[:, :3], accp[:, 3], nnb, o, f"stalled {stalled}")
