"""The far-field pass and the modes that read its lists with NaN, infinite and
overflowing superparticles: walks that do not list the source keep their results
bit for bit, and in the others the pass leaves the source to the pairs, so that
the same values are finite as with pairs alone (a softening of 1e-150 turns the
pass off and leaves the FP32 pair arithmetic as it is)."""
from __future__ import annotations

import numpy as np
import pytest

from petar_gb300 import gpuforce
from petar_gb300.walks import WalkBatch

pytestmark = pytest.mark.gpu

N_W, N_I, N_S = 24, 400, 4600


def _batch() -> WalkBatch:
    rng = np.random.default_rng(12)
    pos = np.repeat(rng.normal(size=(N_W, 3)), N_I, axis=0) + rng.uniform(-0.05, 0.05, (N_W * N_I, 3))
    n_j, n_src = 2000, N_S + 1
    walk = np.arange(N_W + 1, dtype=np.int64)
    # source 0 in the lists of every second walk, in the place of source 1
    ids = np.stack([1 + rng.permutation(N_S) for _ in range(N_W)])
    ids[::2][ids[::2] == 1] = 0
    return WalkBatch(epi_pos=pos, epi_rs=np.full(N_W * N_I, 0.03), epi_disp=walk * N_I,
                     epj_pos=rng.normal(size=(n_j, 3)), epj_mass=rng.uniform(0.1, 1, n_j) / n_j,
                     epj_rs=np.full(n_j, 0.03), spj_pos=rng.normal(size=(n_src, 3)) * 5,
                     spj_mass=rng.uniform(0.1, 1, n_src) / n_src, spj_quad=rng.normal(size=(n_src, 6)) * 1e-6,
                     epj_disp=walk * 300, id_epj=rng.integers(0, n_j, N_W * 300).astype(np.int32),
                     spj_disp=walk * N_S, id_spj=ids.reshape(-1).astype(np.int32), eps2=0.0, rcut2=0.02 ** 2, G=1.0)


def _run(wb, mode):
    if mode == "gradient":
        rng = np.random.default_rng(1)
        f = gpuforce.compute_gradient(wb, rng.normal(size=wb.epi_pos.shape), rng.normal(size=wb.epj_pos.shape))
    else:
        f = gpuforce.compute(wb)
    return np.concatenate([f["acc"], f["pot"][:, None]], axis=1).reshape(N_W, N_I, 4)


@pytest.mark.parametrize("mode", ["force", "gradient"])
@pytest.mark.parametrize("field,value", [("pos", np.nan), ("pos", np.inf), ("pos", -1e300), ("pos", 1e25),
                                         ("mass", np.nan), ("mass", np.inf), ("mass", 1e35), ("mass", -1e300),
                                         ("quad", np.nan), ("quad", -np.inf), ("quad", 1e38)])
def test_special_source(mode, field, value):
    wb = _batch()
    clean = _run(wb, mode)
    assert np.isfinite(clean).all()
    if field == "pos":
        wb.spj_pos[0, 1] = value
    elif field == "mass":
        wb.spj_mass[0] = value
    else:
        wb.spj_quad[0, 2] = value
    got = _run(wb, mode)
    np.testing.assert_array_equal(got[1::2], clean[1::2])
    wb.eps2 = 1e-300
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(_run(wb, mode)))
