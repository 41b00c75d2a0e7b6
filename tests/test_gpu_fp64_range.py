"""The plain FP64 kernel with sources so far away that r^2 is beyond FP64's
range: 1/r is 0 there, as in the oracle, and they add nothing.  Same bound as
the other edges of this kernel: 6.3e-13 of the sum of the terms' magnitudes.
And with a NaN coordinate of an EPJ: the clamp to r_out takes an unordered r^2
for one inside it, so that the NaN reaches that coordinate of the acceleration
of its walk's i and nothing else."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from petar_gb300 import gpuforce
from petar_gb300.walks import WalkBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e154, 1e160, 1e250])
def test_sources_beyond_the_range_of_r2(far):
    rng = np.random.default_rng(2)
    n_i, n_j, n_s = 70, 300, 300
    pos = rng.normal(size=(n_i, 3)) * 0.1
    ej, sj = rng.normal(size=(n_j, 3)), rng.normal(size=(n_s, 3)) + 3.0
    ej[::50], sj[::50] = far, -far
    q = rng.normal(size=(n_s, 6)) * 0.01
    q[::50] = 0.0
    disp = lambda n: np.array([0, n], np.int64)
    wb = WalkBatch(epi_pos=pos, epi_rs=np.full(n_i, 0.03), epi_disp=disp(n_i), epj_pos=ej,
                   epj_mass=rng.uniform(0, 1, n_j), epj_rs=np.full(n_j, 0.03), spj_pos=sj,
                   spj_mass=rng.uniform(0, 1, n_s), spj_quad=q, epj_disp=disp(n_j),
                   id_epj=np.arange(n_j, dtype=np.int32), spj_disp=disp(n_s), id_spj=np.arange(n_s, dtype=np.int32),
                   eps2=0.0, rcut2=0.02 ** 2, G=1.0)
    try:
        f = gpuforce.compute(wb, gpuforce.PGF_PRECISION_FP64)
    finally:
        gpuforce.set_precision(gpuforce.PGF_PRECISION_MIXED)
    with np.errstate(over="ignore"):
        o = oracle.force(wb)
    mag = np.zeros(n_i)
    for x, m in ((ej, wb.epj_mass), (sj, wb.spj_mass)):
        near = np.abs(x).max(1) < 1e3
        d2 = np.maximum(((x[near][None] - pos[:, None]) ** 2).sum(-1), wb.rcut2)
        mag += (m[near] / d2).sum(1)
    assert np.isfinite(o["acc"]).all() and np.isfinite(o["pot"]).all()
    np.testing.assert_array_equal(f["nnb"], o["nnb"])
    assert (np.linalg.norm(f["acc"] - o["acc"], axis=1) <= 6.3e-13 * mag).all()
    assert (np.abs(f["pot"] - o["pot"]) <= 6.3e-13 * np.maximum(np.abs(o["pot"]), mag)).all()


def test_nan_coordinate_reaches_its_component_alone():
    rng = np.random.default_rng(5)
    n_w, n_i, n_j = 6, 80, 400
    pos = rng.normal(size=(n_w * n_i, 3)) * 0.1
    ej = rng.normal(size=(n_w * n_j, 3)) * 2.0
    walk = np.arange(n_w + 1, dtype=np.int64)
    wb = WalkBatch(epi_pos=pos, epi_rs=np.full(n_w * n_i, 0.03), epi_disp=walk * n_i, epj_pos=ej,
                   epj_mass=rng.uniform(0, 1, n_w * n_j), epj_rs=np.full(n_w * n_j, 0.03),
                   spj_pos=np.full((1, 3), 9.0), spj_mass=np.ones(1), spj_quad=np.zeros((1, 6)), epj_disp=walk * n_j,
                   id_epj=np.arange(n_w * n_j, dtype=np.int32), spj_disp=walk * 0, id_spj=np.zeros(0, np.int32),
                   eps2=0.0, rcut2=0.02 ** 2, G=1.0)
    bad = {0: 0, 2: 1, 4: 2}  # walk: coordinate
    for w, c in bad.items():
        ej[w * n_j + 17 * (w + 1), c] = np.nan
    try:
        f = gpuforce.compute(wb, gpuforce.PGF_PRECISION_FP64)
    finally:
        gpuforce.set_precision(gpuforce.PGF_PRECISION_MIXED)
    want = np.ones((n_w * n_i, 3), bool)
    for w, c in bad.items():
        want[w * n_i:(w + 1) * n_i, c] = False
    np.testing.assert_array_equal(np.isfinite(f["acc"]), want)
    assert np.isfinite(f["pot"]).all()
