"""Device memory of a device-resident handle in small clusters: result rows for
the parts of split walks and re-test records in proportion to what it can use.
A walk of 700 stars has at most 31 further parts, so the rows take at most
31 x 700 x 36 bytes; everything else is a few hundred bytes a particle.  The
driver hands out device memory in units of 2 MB, one of them for all small
arrays of a kind here: 24 MB is far above the need and well below the 70 MB
that rows and records for the largest clusters take."""
from __future__ import annotations

import pytest

from petar_gb300 import gpuforce, ics, nbody

pytestmark = pytest.mark.gpu


def test_small_handles_stay_small():
    torch = pytest.importorskip("torch")
    cl = ics.make_king_cluster(2, 700, 0.02, W0=6.0, theta=0.5)
    with nbody.DeviceNBody(cl) as h:  # loads the kernels
        h.run(1, 0.0)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with nbody.DeviceNBody(cl) as h:
        used = free - torch.cuda.mem_get_info()[0]
        want = h.state()
    assert used <= 24 << 20, used
    # the kernel that needs the records has them, also when it is tried later
    with nbody.DeviceNBody(cl, kernel_variant=0) as h:
        got = h.state()
        assert (got["n_ngb"] == want["n_ngb"]).all()
    with nbody.DeviceNBody(cl) as h:
        h.autotune(1)
        assert (h.state()["n_ngb"] == want["n_ngb"]).all()
    assert gpuforce.get_kernel_variant() != 0
