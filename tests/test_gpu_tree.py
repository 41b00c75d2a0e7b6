"""Device tree where its moments run a cell per lane (more cells of a class
than a grid of 8-lane groups holds) and a few shares more or fewer than the
CTAs take at a time, and lists on both sides of the top pass's line (131,072
particles): lists and moments against the host builder, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from petar_gb300 import ics, nbody, walks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_leaf", [(57001, 8), (40009, 2), (131071, 8), (131072, 8), (260003, 20)])
def test_tree_equals_host_builder(n, n_leaf):
    cl = ics.make_king_cluster(9, n, 0.004, W0=6.0, theta=0.5)
    cl.n_leaf_limit = n_leaf
    host = walks.build_walks(cl)
    with nbody.DeviceNBody(cl) as h:
        dev = h.lists()
        cells = h.stats()["n_cells"]
    assert cells > 9728  # 152 CTAs x 512 lanes / 8
    for k in ("epi_index", "epi_disp", "epj_disp", "spj_disp", "id_epj", "id_spj", "spj_mass", "spj_pos", "spj_quad"):
        np.testing.assert_array_equal(getattr(dev, k), getattr(host, k), err_msg=k)
