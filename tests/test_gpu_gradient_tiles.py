"""Gradient pass at the edges of its tiles (256 entries) and passes (512 i of
a walk at a time): every component against the FP64 oracle within 1e-6 of the
sum of its terms' magnitudes (a term's chain of about 16 FP32 roundings of
2^-24 each)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from petar_gb300 import gpuforce
from petar_gb300.walks import WalkBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_i,n_epj,n_spj", [
    ([1, 255, 513, 1030], [255, 256, 257, 513], [0, 1, 256, 257]),
    ([511, 1025, 2, 700], [768, 1, 0, 511], [255, 512, 513, 0]),
])
def test_gradient_tiles(n_i, n_epj, n_spj):
    rng = np.random.default_rng(5)
    disp = lambda v: np.concatenate([[0], np.cumsum(v)]).astype(np.int64)
    nw, ni, nj, ns = len(n_i), sum(n_i), 900, 600
    pos = np.repeat(rng.normal(size=(nw, 3)), n_i, axis=0) + rng.uniform(-0.1, 0.1, (ni, 3))
    wb = WalkBatch(epi_pos=pos, epi_rs=np.full(ni, 0.03), epi_disp=disp(n_i), epj_pos=rng.normal(size=(nj, 3)),
                   epj_mass=rng.uniform(0.1, 1, nj) / nj, epj_rs=np.full(nj, 0.03),
                   spj_pos=rng.normal(size=(ns, 3)) * 2 + 6.0, spj_mass=rng.uniform(0.1, 1, ns) / ns,
                   spj_quad=rng.normal(size=(ns, 6)) * 1e-6, epj_disp=disp(n_epj),
                   id_epj=rng.integers(0, nj, sum(n_epj)).astype(np.int32), spj_disp=disp(n_spj),
                   id_spj=rng.integers(0, ns, sum(n_spj)).astype(np.int32), eps2=0.0, rcut2=0.1 ** 2, G=1.0)
    ai, aj = rng.normal(size=(ni, 3)), rng.normal(size=(nj, 3))
    o = oracle.gradient(wb, ai, aj)
    mag, amag = np.zeros(ni), np.linalg.norm(ai, axis=1)
    for w in range(nw):
        for i in range(wb.epi_disp[w], wb.epi_disp[w + 1]):
            ids = wb.id_epj[wb.epj_disp[w]:wb.epj_disp[w + 1]]
            r = np.maximum(np.linalg.norm(wb.epj_pos[ids] - pos[i], axis=1), 0.1)
            da = np.linalg.norm(aj[ids] - ai[i], axis=1)
            mag[i] = 2 * np.sum(wb.epj_mass[ids] * 4 * da / r ** 3)
            sid = wb.id_spj[wb.spj_disp[w]:wb.spj_disp[w + 1]]
            amag[i] += np.sum(wb.spj_mass[sid] / np.sum((wb.spj_pos[sid] - pos[i]) ** 2, axis=1))
    for _ in range(3):
        res = gpuforce.compute_gradient(wb, ai, aj)
        assert (np.linalg.norm(res["acorr"] - o["acorr"], axis=1) <= 1e-6 * mag).all()
        assert (np.linalg.norm(res["acc"] - o["acc"], axis=1) <= 1e-6 * amag).all()
        assert (res["nnb"] == 0).all()
