"""The far-field pass on walks whose distant sources all lie on one side, where
nothing averages its truncation out: the force must be as good as that of the
pairs.  A softening of 1e-150 turns the pass off and leaves the FP32 pair
arithmetic as it is, so the same call gives the pairs' error.

The pass may add 2^-23 of the sum of the sources' force magnitudes by
truncation (its limit for a source) and as much again by rounding: rows 2 and
up of the expansion are at most rho = 0.14 of the leading ones and carry about
ten FP32 roundings each."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from petar_gb300 import gpuforce
from petar_gb300.walks import WalkBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [8192, 40960])  # eight warps per walk, and four
@pytest.mark.parametrize("near,far,quad", [(7.2, 7.4, 0.0), (7.2, 8.5, 3e-4), (7.5, 30.0, 0.0), (7.2, 400.0, 1e-4),
                                           (10.02, 10.3, 0.0), (10.5, 16.0, 1e-4)])
def test_one_sided_sources(rows, near, far, quad):
    rng = np.random.default_rng(3)
    n_i, n_s, R = 64, 4200, 0.1
    nw = rows // n_i
    u = rng.normal(size=(nw, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    cen = rng.normal(size=(nw, 3))
    # i on the sphere of radius R, half of them close to the sources' direction; +-u keeps the box's centre
    x = rng.normal(size=(nw, n_i, 3)) * 0.3
    x[:, : n_i // 2] += u[:, None]
    x *= R / np.linalg.norm(x, axis=2)[:, :, None]
    x[:, 0], x[:, 1] = R * u, -R * u
    lo, hi = x.min(1), x.max(1)
    x -= (0.5 * (lo + hi))[:, None]
    r_w = np.linalg.norm(x, axis=2).max(1)  # each walk's radius about its box's centre
    pos = (cen[:, None] + x).reshape(-1, 3)
    e = rng.normal(size=(nw, n_s, 3)) * 0.05 + u[:, None]
    e /= np.linalg.norm(e, axis=2)[:, :, None]
    D = r_w[:, None] * np.exp(rng.uniform(np.log(near), np.log(far), (nw, n_s)))
    spos = (cen[:, None] + e * D[:, :, None]).reshape(-1, 3)
    m = rng.uniform(0.5, 1.0, nw * n_s)
    q = rng.normal(size=(nw * n_s, 6)) * (quad * m * D.reshape(-1) ** 2)[:, None]
    disp_i = np.arange(nw + 1, dtype=np.int64) * n_i
    wb = WalkBatch(epi_pos=pos, epi_rs=np.full(pos.shape[0], 0.01), epi_disp=disp_i, epj_pos=pos[:1] + 50.0,
                   epj_mass=np.full(1, 1e-9), epj_rs=np.full(1, 0.01), spj_pos=spos, spj_mass=m, spj_quad=q,
                   epj_disp=np.zeros(nw + 1, np.int64), id_epj=np.zeros(0, np.int32),
                   spj_disp=np.arange(nw + 1, dtype=np.int64) * n_s, id_spj=np.arange(nw * n_s, dtype=np.int32),
                   eps2=0.0, rcut2=1e-4, G=1.0)
    own = wb.subset(np.arange(64))  # those compared
    n = own.epi_rs.size
    with_pass = gpuforce.compute(wb)
    o = oracle.force(own)
    wb.eps2 = 1e-300
    pairs = gpuforce.compute(wb)
    mag = np.linalg.norm(o["acc"], axis=1)  # one side: the sum of the magnitudes, to the spread of 0.05
    err = lambda f: np.linalg.norm(f["acc"][:n] - o["acc"], axis=1) / mag
    ef, ep = err(with_pass), err(pairs)
    assert ef.max() <= ep.max() + 2 * 2.0 ** -23, (ef.max(), ep.max())
    assert ef.mean() <= ep.mean() + 2.0 ** -23, (ef.mean(), ep.mean())
    pf, pp = (np.abs(f["pot"][:n] - o["pot"]) / np.abs(o["pot"]) for f in (with_pass, pairs))
    assert pf.max() <= pp.max() + 2 * 2.0 ** -23, (pf.max(), pp.max())
