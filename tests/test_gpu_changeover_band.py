"""Changeover mode, pairs inside the guard band of the neighbour test (r_search
to a few FP32 roundings): whether such a pair is a neighbour is decided in FP64,
and what that changes is added as computed in FP64.  For companions deep inside
the changeover the potential -m / r is far larger than the linear cutoff's
m / r_out that FP32 carries, so its error is that part's: a reciprocal square
root (2^-22.9) and three roundings (2^-24) of m / r_out, and 2^-44 of the sums."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from petar_gb300 import gpuforce, walks
from petar_gb300.walks import WalkBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rs,n_j", [(1e-4, 1), (1e-5, 1), (1e-5, 3)])
def test_companions_at_the_search_radius(rs, n_j):
    rng = np.random.default_rng(1)
    n, r_in, r_out = 4000, 0.001, 0.0093
    x = rng.normal(size=(n, 3)) * 1e-3
    u = rng.normal(size=(n, n_j, 3))
    u /= np.linalg.norm(u, axis=2)[:, :, None]
    r = rs * (1 + rng.uniform(-3e-7, 3e-7, (n, n_j)))
    ej = (x[:, None] + u * r[:, :, None]).reshape(-1, 3)
    m = rng.uniform(0.5, 1.5, n * n_j).astype(np.float32).astype(float)  # as the records hold them
    d = np.arange(n + 1, dtype=np.int64)
    wb = WalkBatch(epi_pos=x, epi_rs=np.full(n, rs), epi_disp=d, epj_pos=ej, epj_mass=m, epj_rs=np.full(n * n_j, rs),
                   spj_pos=x[:1] + 9.0, spj_mass=np.ones(1), spj_quad=np.zeros((1, 6)), epj_disp=d * n_j,
                   id_epj=np.arange(n * n_j, dtype=np.int32), spj_disp=d * 0, id_spj=np.zeros(0, np.int32),
                   eps2=0.0, rcut2=r_out ** 2, G=1.0)
    one = np.ones(n * n_j)
    co = walks.ChangeoverSet(np.arange(n, dtype=np.int64), np.full(n, r_in), np.full(n, r_out), np.zeros(n),
                             n + np.arange(n * n_j, dtype=np.int64), r_in * one, r_out * one, 0 * one, 0 * one)
    f, o = gpuforce.compute_changeover(wb, co), oracle.force_changeover(wb, co)
    np.testing.assert_array_equal(f["nnb"], o["nnb"])
    neighbours = o["nnb"] == n_j
    assert 0.1 < neighbours.mean() < 0.9
    cutoff = m.reshape(n, n_j).sum(1) / r_out
    tol = cutoff * (2.0 ** -22.9 + 3 * 2.0 ** -24) + 2.0 ** -44 * np.abs(o["pot"])
    err = np.abs(f["pot"] - o["pot"])
    assert (err[neighbours] <= tol[neighbours]).all(), (err / tol)[neighbours].max()
