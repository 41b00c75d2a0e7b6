"""The far-field pass at the edges of test_gpu_far.py in each of its two
kernels and in the modes that read its compacted lists.  Walks of 2,048 i with
lists of 5,300 bring a dispatch to the pass: five of them to the kernel with
eight warps per walk, twenty to the one with four.  The case's own walks are
compared with the oracle; the bound is that test's: 4e-6 of the sum of the
sources' force magnitudes by truncation at most (the pass keeps well below),
2e-6 by FP32 arithmetic."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import test_gpu_far as far
from petar_gb300 import gpuforce, walks

pytestmark = pytest.mark.gpu


def _batch(warps, name):
    """The dispatch, its first walks alone (those of the case), and the bounds of their rows."""
    case = dict(far.CASES[name])
    n, big = len(case["n_i"]), 20 if warps == 4 else 5
    case.update(n_i=case["n_i"] + [2048] * big, n_spj=case["n_spj"] + [5300] * big)
    wb = far._batch(7, **case)
    rows = wb.epi_rs.size
    assert int((wb.n_epi * wb.n_spj).sum()) >= 4000 * rows and (8192 <= rows <= 40000 if warps == 8 else rows > 40000)
    own = wb.subset(np.arange(n))
    mag, pot = far._magnitudes(own)
    scale = 6e-6 * (1.0 + 6.0 * case.get("quad", 0.02))
    return wb, own, scale * mag + 1e-30, scale * pot + 1e-30


@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("name", sorted(far.CASES))
@pytest.mark.parametrize("split", [False, True])
def test_force_mode(warps, name, split):
    wb, own, tol, tol_pot = _batch(warps, name)
    gpuforce.set_walk_split(split)
    try:
        f = gpuforce.compute(wb)
    finally:
        gpuforce.set_walk_split(True)
    o, n = oracle.force(own), tol.size
    assert (np.linalg.norm(f["acc"][:n] - o["acc"], axis=1) <= tol).all()
    assert (np.abs(f["pot"][:n] - o["pot"]) <= tol_pot).all()
    np.testing.assert_array_equal(f["nnb"][:n], o["nnb"])


@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("name", sorted(far.CASES))
def test_changeover_mode(warps, name):
    wb, own, tol, tol_pot = _batch(warps, name)
    n, one = wb.epi_rs.size, np.ones(1)
    # no self-potential: the bound is about the sources'
    co = walks.ChangeoverSet(np.arange(n, dtype=np.int64), np.full(n, 0.001), np.full(n, 0.01), np.zeros(n),
                             np.full(1, n, np.int64), 0.001 * one, 0.01 * one, 0 * one, 0 * one)
    f = gpuforce.compute_changeover(wb, co)
    o, n = oracle.force_changeover(own, walks.subset_changeover(wb, co, np.arange(own.n_walk))), tol.size
    assert (np.linalg.norm(f["acc"][:n] - o["acc"], axis=1) <= tol).all()
    for k in ("pot", "pot_soft"):
        assert (np.abs(f[k][:n] - o[k]) <= tol_pot).all()
    np.testing.assert_array_equal(f["nnb"][:n], o["nnb"])


@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("name", sorted(far.CASES))
@pytest.mark.parametrize("compensated", [0, 1])
def test_gradient_mode(warps, name, compensated):
    wb, own, tol, tol_pot = _batch(warps, name)
    zero = np.zeros((wb.epi_rs.size, 3)), np.zeros((wb.epj_rs.size, 3))
    gpuforce.set_gradient_accuracy(compensated)
    try:
        f = gpuforce.compute_gradient(wb, *zero)
    finally:
        gpuforce.set_gradient_accuracy(1)
    n = tol.size
    o = oracle.gradient(own, zero[0][:n], zero[1])
    assert (np.linalg.norm(f["acc"][:n] - o["acc"], axis=1) <= tol).all()
    assert (np.abs(f["pot"][:n] - o["pot"]) <= tol_pot).all()
    assert (f["acorr"] == 0).all()
