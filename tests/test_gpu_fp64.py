"""The plain FP64 kernel at the edges of its passes, slices and tiles, and at
the border between its far and near pairs, against the FP64 oracle.

Both sum the same terms in FP64 in another order: with at most 1,400 terms of
a few ulp each the difference stays below 1,400 x 4 x 2^-53 = 6.3e-13 of the
sum of the terms' magnitudes, and typically far below."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from petar_gb300 import gpuforce
from petar_gb300.walks import WalkBatch

pytestmark = pytest.mark.gpu


def _batch(seed: int, n_i: list, n_epj: list, n_spj: list, eps2: float) -> WalkBatch:
    rng = np.random.default_rng(seed)
    nw, ni, n_j, n_s = len(n_i), sum(n_i), 900, 500
    disp = lambda c: np.concatenate([[0], np.cumsum(c)]).astype(np.int64)
    # particles close to and far from the walks, some at r_out and r_search to rounding, one on an i
    pos = rng.normal(size=(ni, 3)) * 0.05
    ej = rng.normal(size=(n_j, 3)) * np.exp(rng.uniform(-4, 2, n_j))[:, None]
    u = rng.normal(size=(30, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    ej[:30] = pos[:30 % ni or 1][0] + u * np.repeat([0.02, 0.03, 0.02 * (1 - 1e-15)], 10)[:, None]
    ej[30] = pos[0]
    q = rng.normal(size=(n_s, 6)) * 0.01
    return WalkBatch(epi_pos=pos, epi_rs=np.full(ni, 0.03), epi_disp=disp(n_i), epj_pos=ej,
                     epj_mass=rng.uniform(0, 1, n_j), epj_rs=rng.choice([0.0, 0.03, 0.05], n_j),
                     spj_pos=rng.normal(size=(n_s, 3)) + 3.0, spj_mass=rng.uniform(0, 1, n_s), spj_quad=q,
                     epj_disp=disp(n_epj), id_epj=rng.integers(0, n_j, sum(n_epj)).astype(np.int32),
                     spj_disp=disp(n_spj), id_spj=rng.integers(0, n_s, sum(n_spj)).astype(np.int32),
                     eps2=eps2, rcut2=0.02 ** 2, G=1.0)


@pytest.mark.parametrize("eps2", [0.0, 1e-6])
@pytest.mark.parametrize("split", [False, True])
def test_fp64_edges(eps2, split):
    n_i = [1, 2, 31, 32, 33, 85, 86, 127, 128, 129, 255, 256, 257, 513]
    n_epj = [900, 1, 255, 256, 257, 0, 512, 100, 300, 900, 700, 256, 511, 700]
    n_spj = [0, 500, 255, 256, 257, 100, 0, 1, 300, 500, 400, 256, 100, 500]
    wb = _batch(3, n_i, n_epj, n_spj, eps2)
    gpuforce.set_walk_split(split)
    try:
        f = gpuforce.compute(wb, gpuforce.PGF_PRECISION_FP64)
    finally:
        gpuforce.set_walk_split(True)
        gpuforce.set_precision(gpuforce.PGF_PRECISION_MIXED)
    o = oracle.force(wb)
    np.testing.assert_array_equal(f["nnb"], o["nnb"])
    mag, pot = np.full(wb.epi_rs.size, 1e-300), np.full(wb.epi_rs.size, 1e-300)
    for w in range(wb.n_walk):
        r = slice(wb.epi_disp[w], wb.epi_disp[w + 1])
        for j, x, m in ((wb.id_epj[wb.epj_disp[w]:wb.epj_disp[w + 1]], wb.epj_pos, wb.epj_mass),
                        (wb.id_spj[wb.spj_disp[w]:wb.spj_disp[w + 1]], wb.spj_pos, wb.spj_mass)):
            d2 = np.maximum(((x[j][None] - wb.epi_pos[r][:, None]) ** 2).sum(-1), wb.rcut2)
            mag[r] += (m[j] / d2).sum(1)
            pot[r] += (m[j] / np.sqrt(d2)).sum(1)
    assert (np.linalg.norm(f["acc"] - o["acc"], axis=1) <= 6.3e-13 * mag).all()
    assert (np.abs(f["pot"] - o["pot"]) <= 6.3e-13 * pot).all()
