"""Walk splitting planned on the device (the allocation-free entry point uses
it on the caller's tables): lists at the edges of the parts, which are cut at
multiples of 256 entries, one walk that dominates the rest, and walks whose
parts would not fit the scratch rows, against the FP64 oracle at the
mixed-precision bar of the parity tests."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from helpers import assert_mixed_parity
from petar_gb300.walks import WalkBatch
from test_zz_no_alloc import _call, _device_inputs, _lib

pytestmark = pytest.mark.gpu

CASES = {
    # list lengths around the parts' grain, i counts around the pass layouts
    "edges": dict(n_i=[300, 385, 129, 64, 1, 500, 33], n_epj=[255, 256, 257, 511, 3000, 0, 512],
                  n_spj=[0, 513, 256, 1, 700, 1025, 255]),
    # one walk holds nearly all the work (32 parts at most), many hold none
    "one_walk": dict(n_i=[450] + [1] * 40, n_epj=[30000] + [3] * 40, n_spj=[9000] + [0] * 40),
    # parts of a sixteenth of an SM's share would need 2,000,000 rows
    "rows": dict(n_i=[2500] * 40, n_epj=[6000] * 40, n_spj=[300] * 40),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_device_plan(name):
    torch = pytest.importorskip("torch")
    c = CASES[name]
    rng = np.random.default_rng(11)
    disp = lambda v: np.concatenate([[0], np.cumsum(v)]).astype(np.int64)
    nw, ni, nj, ns = len(c["n_i"]), sum(c["n_i"]), 4000, 1000
    cen = rng.normal(size=(nw, 3))
    pos = np.repeat(cen, c["n_i"], axis=0) + rng.uniform(-0.1, 0.1, (ni, 3))
    q = rng.normal(size=(ns, 6)) * 1e-6
    wb = WalkBatch(epi_pos=pos, epi_rs=np.full(ni, 0.03), epi_disp=disp(c["n_i"]), epj_pos=rng.normal(size=(nj, 3)),
                   epj_mass=rng.uniform(0.1, 1, nj) / nj, epj_rs=np.full(nj, 0.03),
                   spj_pos=rng.normal(size=(ns, 3)) * 2 + 6.0, spj_mass=rng.uniform(0.1, 1, ns) / ns, spj_quad=q,
                   epj_disp=disp(c["n_epj"]), id_epj=rng.integers(0, nj, sum(c["n_epj"])).astype(np.int32),
                   spj_disp=disp(c["n_spj"]), id_spj=rng.integers(0, ns, sum(c["n_spj"])).astype(np.int32),
                   eps2=0.0, rcut2=0.02 ** 2, G=1.0)
    f, d = _lib(), _device_inputs(torch, wb)
    for _ in range(2):  # the scratch is shared by all calls
        _call(f, torch, wb, d)
        torch.cuda.synchronize()
        a, n = d["accp"].cpu().numpy(), d["nnb"].cpu().numpy()
        o = oracle.force(wb)
        has = np.repeat(np.asarray(c["n_epj"]) + np.asarray(c["n_spj"]) > 0, c["n_i"])
        assert_mixed_parity(a[has, :3], a[has, 3], n[has], {k: o[k][has] for k in ("acc", "pot", "nnb")}, name)
        assert (a[~has] == 0).all() and (n[~has] == 0).all()
