"""The far-field pass (local expansions of distant superparticles): walks whose
lists sit at its edges against the FP64 oracle.

A source is expanded when the dropped terms stay below 2e-6 of its own force
for the monopole and for the quadrupole each, so a walk's error is at most
4e-6 of the sum of its sources' force magnitudes; FP32 pair arithmetic and
sums add less than 2e-6 of that sum (about 30 roundings of 2^-24)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from petar_gb300 import gpuforce
from petar_gb300.walks import WalkBatch

pytestmark = pytest.mark.gpu

ROWS = 8192  # the pass runs from this many i-particles per launch


def _batch(seed: int, n_i: list, n_spj: list, near: float, far: float, centre=0.0, quad=0.02) -> WalkBatch:
    """Walks of radius about 0.1 with sources at log-uniform distances between
    near and far from their centres, padded with small walks to ROWS rows."""
    rng = np.random.default_rng(seed)
    n_i, n_spj = list(n_i), list(n_spj)
    while sum(n_i) < ROWS:
        n_i.append(31)
        n_spj.append(3)
    nw = len(n_i)
    disp = lambda c: np.concatenate([[0], np.cumsum(c)]).astype(np.int64)
    ei, es = disp(n_i), disp(n_spj)
    cen = centre + rng.normal(size=(nw, 3))
    pos = np.repeat(cen, n_i, axis=0) + rng.uniform(-0.06, 0.06, (ei[-1], 3))
    d = rng.normal(size=(es[-1], 3))
    d *= (np.exp(rng.uniform(np.log(near), np.log(far), es[-1])) / np.linalg.norm(d, axis=1))[:, None]
    m = rng.uniform(0.1, 1.0, es[-1]) * 1e-3
    m[::17] = 0.0  # massless sources without moments
    q = rng.normal(size=(es[-1], 6)) * (quad * m * (d * d).sum(1))[:, None]
    order = rng.permutation(es[-1])  # the lists are gathers
    spos, sm, sq = np.empty_like(d), np.empty_like(m), np.empty_like(q)
    spos[order] = np.repeat(cen, n_spj, axis=0) + d
    sm[order], sq[order] = m, q
    return WalkBatch(epi_pos=pos, epi_rs=np.full(ei[-1], 0.01), epi_disp=ei, epj_pos=pos[:1] + 50.0,
                     epj_mass=np.full(1, 1e-9), epj_rs=np.full(1, 0.01), spj_pos=spos, spj_mass=sm, spj_quad=sq,
                     epj_disp=np.zeros(nw + 1, np.int64), id_epj=np.zeros(0, np.int32), spj_disp=es,
                     id_spj=order.astype(np.int32), eps2=0.0, rcut2=1e-4, G=1.0)


def _magnitudes(wb: WalkBatch) -> tuple:
    """Sums over each row's sources of the monopole force and potential magnitudes."""
    out, pot = np.zeros(wb.epi_rs.size), np.zeros(wb.epi_rs.size)
    for w in range(wb.n_walk):
        j = wb.id_spj[wb.spj_disp[w]:wb.spj_disp[w + 1]]
        r = slice(wb.epi_disp[w], wb.epi_disp[w + 1])
        d = wb.spj_pos[j][None] - wb.epi_pos[r][:, None]
        r2 = (d * d).sum(-1)
        out[r] = (wb.spj_mass[j][None] / r2).sum(1)
        pot[r] = (wb.spj_mass[j][None] / np.sqrt(r2)).sum(1)
    return out, pot


CASES = {
    # i counts around the pass's least (32) and a warp, list lengths around a lane group and a quarter
    "edges": dict(n_i=[31, 32, 33, 64, 127, 128, 129, 300], n_spj=[200, 1, 31, 32, 33, 127, 129, 1000], near=0.5, far=20.0),
    # every source distant, every source close, and none
    "all_far": dict(n_i=[40, 100, 200], n_spj=[5, 128, 515], near=3.0, far=1000.0),
    "none_far": dict(n_i=[40, 100, 200], n_spj=[5, 128, 515], near=0.2, far=0.5),
    "empty": dict(n_i=[40, 100], n_spj=[0, 0], near=1.0, far=2.0),
    # more i than one pass and than the coordinates kept in shared memory
    "large": dict(n_i=[511, 512, 513, 1500], n_spj=[700, 701, 702, 703], near=0.5, far=50.0),
    # lists whose half quarters are longer than the pass keeps in shared memory
    "long": dict(n_i=[64, 100], n_spj=[16390, 17000], near=0.5, far=50.0),
    # walks away from the origin (x - c cancels), large moments
    "offset": dict(n_i=[64, 200], n_spj=[400, 3000], near=0.5, far=20.0, centre=300.0),
    "moments": dict(n_i=[64, 200], n_spj=[400, 3000], near=0.5, far=20.0, quad=2.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("split", [False, True])
def test_far_pass_against_oracle(name, split):
    wb = _batch(7, **CASES[name])
    gpuforce.set_walk_split(split)
    try:
        f = gpuforce.compute(wb)
    finally:
        gpuforce.set_walk_split(True)
    o = oracle.force(wb)
    mag, mag_pot = _magnitudes(wb)
    scale = 1.0 + 6.0 * CASES[name].get("quad", 0.02)  # quadrupole forces next to the monopole's
    err = np.linalg.norm(f["acc"] - o["acc"], axis=1)
    assert (err <= 6e-6 * scale * mag + 1e-30).all(), (err / np.maximum(mag, 1e-300)).max()
    assert (np.abs(f["pot"] - o["pot"]) <= 6e-6 * scale * mag_pot + 1e-30).all()
    np.testing.assert_array_equal(f["nnb"], o["nnb"])


def test_far_pass_is_deterministic_and_off_when_softened():
    wb = _batch(8, **CASES["edges"])
    a, b = gpuforce.compute(wb), gpuforce.compute(wb)
    np.testing.assert_array_equal(a["acc"], b["acc"])
    wb.eps2 = 1e-4  # softened gravity: pairs only
    f, o = gpuforce.compute(wb), oracle.force(wb)
    assert (np.linalg.norm(f["acc"] - o["acc"], axis=1) <= 2e-6 * _magnitudes(wb)[0] + 1e-30).all()
