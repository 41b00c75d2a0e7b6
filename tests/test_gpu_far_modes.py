"""The far-field pass at the edges of test_gpu_far.py in each of its two
kernels and in the modes that read its compacted lists.  Dispatches of many
i-particles run the kernel with four warps per walk, those of few with long
lists the one with eight; small walks and walks of 2,048 i with lists of 5,300
make the cases' dispatches the one or the other.  The bound is that test's:
4e-6 of the sum of the sources' force magnitudes by truncation at most (the
pass keeps well below), 2e-6 by FP32 arithmetic."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import test_gpu_far as far
from petar_gb300 import gpuforce, walks

pytestmark = pytest.mark.gpu


def _magnitudes(wb):
    f, pot = np.zeros(wb.epi_rs.size), np.zeros(wb.epi_rs.size)
    for w in range(wb.n_walk):
        j = wb.id_spj[wb.spj_disp[w]:wb.spj_disp[w + 1]]
        for r0 in range(int(wb.epi_disp[w]), int(wb.epi_disp[w + 1]), 128):
            r = slice(r0, min(r0 + 128, int(wb.epi_disp[w + 1])))
            d2 = ((wb.spj_pos[j][None] - wb.epi_pos[r][:, None]) ** 2).sum(-1)
            f[r] = (wb.spj_mass[j][None] / d2).sum(1)
            pot[r] = (wb.spj_mass[j][None] / np.sqrt(d2)).sum(1)
    return f, pot


def _batch(monkeypatch, warps, name):
    case = dict(far.CASES[name])
    if warps == 4:
        monkeypatch.setattr(far, "ROWS", 80001)
    else:
        case.update(n_i=case["n_i"] + [2048] * 5, n_spj=case["n_spj"] + [5300] * 5)
    wb = far._batch(7, **case)
    rows, pairs = wb.epi_rs.size, int((wb.n_epi * wb.n_spj).sum())
    assert rows > 80000 if warps == 4 else 8192 <= rows <= 40000 and pairs >= 4000 * rows
    mag, pot = _magnitudes(wb)
    scale = 6e-6 * (1.0 + 6.0 * case.get("quad", 0.02))
    return wb, scale * mag + 1e-30, scale * pot + 1e-30


@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("name", sorted(far.CASES))
@pytest.mark.parametrize("split", [False, True])
def test_force_mode(monkeypatch, warps, name, split):
    wb, tol, tol_pot = _batch(monkeypatch, warps, name)
    gpuforce.set_walk_split(split)
    try:
        f = gpuforce.compute(wb)
    finally:
        gpuforce.set_walk_split(True)
    o = oracle.force(wb)
    assert (np.linalg.norm(f["acc"] - o["acc"], axis=1) <= tol).all()
    assert (np.abs(f["pot"] - o["pot"]) <= tol_pot).all()
    np.testing.assert_array_equal(f["nnb"], o["nnb"])


@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("name", sorted(far.CASES))
def test_changeover_mode(monkeypatch, warps, name):
    wb, tol, tol_pot = _batch(monkeypatch, warps, name)
    n, one = wb.epi_rs.size, np.ones(1)
    # no self-potential: the bound is about the sources'
    co = walks.ChangeoverSet(np.arange(n, dtype=np.int64), np.full(n, 0.001), np.full(n, 0.01), np.zeros(n),
                             np.full(1, n, np.int64), 0.001 * one, 0.01 * one, 0 * one, 0 * one)
    f, o = gpuforce.compute_changeover(wb, co), oracle.force_changeover(wb, co)
    assert (np.linalg.norm(f["acc"] - o["acc"], axis=1) <= tol).all()
    for k in ("pot", "pot_soft"):
        assert (np.abs(f[k] - o[k]) <= tol_pot).all()
    np.testing.assert_array_equal(f["nnb"], o["nnb"])


@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("name", sorted(far.CASES))
@pytest.mark.parametrize("compensated", [0, 1])
def test_gradient_mode(monkeypatch, warps, name, compensated):
    wb, tol, tol_pot = _batch(monkeypatch, warps, name)
    zero = np.zeros((wb.epi_rs.size, 3)), np.zeros((wb.epj_rs.size, 3))
    gpuforce.set_gradient_accuracy(compensated)
    try:
        f = gpuforce.compute_gradient(wb, *zero)
    finally:
        gpuforce.set_gradient_accuracy(1)
    o = oracle.gradient(wb, *zero)
    assert (np.linalg.norm(f["acc"] - o["acc"], axis=1) <= tol).all()
    assert (np.abs(f["pot"] - o["pot"]) <= tol_pot).all()
    assert (f["acorr"] == 0).all()
