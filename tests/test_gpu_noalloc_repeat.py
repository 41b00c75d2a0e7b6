"""The allocation-free entry point with several walks over the same EPI rows
(each writes the rows' results; here they agree, so the rows must hold that
result whichever writes last), split into parts and whole."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from helpers import assert_mixed_parity
from petar_gb300.walks import WalkBatch
from test_zz_no_alloc import _call, _device_inputs, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_i,n_epj,n_spj,times", [(400, 20000, 3000, 8), (3, 100, 10, 5), (700, 9000, 0, 40), (60, 1024, 0, 1000)])
def test_walks_over_the_same_rows(n_i, n_epj, n_spj, times):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(6)
    disp = lambda n: np.array([0, n], np.int64)
    nj, ns = 3000, 800
    wb = WalkBatch(epi_pos=rng.uniform(-0.1, 0.1, (n_i, 3)), epi_rs=np.full(n_i, 0.03), epi_disp=disp(n_i),
                   epj_pos=rng.normal(size=(nj, 3)), epj_mass=rng.uniform(0.1, 1, nj) / nj, epj_rs=np.full(nj, 0.03),
                   spj_pos=rng.normal(size=(ns, 3)) * 2 + 6.0, spj_mass=rng.uniform(0.1, 1, ns) / ns,
                   spj_quad=rng.normal(size=(ns, 6)) * 1e-6, epj_disp=disp(n_epj),
                   id_epj=rng.integers(0, nj, n_epj).astype(np.int32), spj_disp=disp(n_spj),
                   id_spj=rng.integers(0, ns, n_spj).astype(np.int32), eps2=0.0, rcut2=0.02 ** 2, G=1.0)
    o = oracle.force(wb)
    f, d = _lib(), _device_inputs(torch, wb, [0] * times)
    for _ in range(5):
        rc, msg, accp, nnb = _call(f, torch, wb, d)
        assert rc == 0, msg
        assert_mixed_parity(accp[:, :3], accp[:, 3], nnb, o, f"{times} times")
