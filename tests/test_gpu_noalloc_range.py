"""The allocation-free entry point on inputs at the ends of FP64's and FP32's
ranges: search radii whose square FP32 cannot hold, and clusters far from the
origin, against the FP64 oracle at the mixed-precision bar of the parity
tests.

In the second, companions 1e-5 apart lie 4e4 from the origin.  FP64 positions
resolve 7e-12 there, so x - c taken in FP64 keeps the separations the caller
gave; split into 48 bits before the subtraction they would be off by 1e-10,
a hundred thousandth of themselves."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from helpers import assert_mixed_parity
from petar_gb300.walks import WalkBatch
from test_zz_no_alloc import _call, _device_inputs, _lib

pytestmark = pytest.mark.gpu


def _run(wb):
    torch = pytest.importorskip("torch")
    rc, msg, accp, nnb = _call(_lib(), torch, wb, _device_inputs(torch, wb))
    assert rc == 0, msg
    return accp[:, :3], accp[:, 3], nnb


@pytest.mark.parametrize("rs", [1.8e19, 1e20, 1e150, np.inf])
def test_search_radius_beyond_fp32(rs):
    rng = np.random.default_rng(4)
    n_i, n_j, n_s = 150, 700, 40
    disp = lambda n: np.array([0, n], np.int64)
    e_rs = np.full(n_i, 0.05)
    e_rs[::3] = rs
    wb = WalkBatch(epi_pos=rng.normal(size=(n_i, 3)) * 0.1, epi_rs=e_rs, epi_disp=disp(n_i),
                   epj_pos=rng.normal(size=(n_j, 3)) * 2, epj_mass=rng.uniform(0.1, 1, n_j),
                   epj_rs=np.full(n_j, 0.05), spj_pos=rng.normal(size=(n_s, 3)) + 8.0,
                   spj_mass=rng.uniform(0.1, 1, n_s), spj_quad=rng.normal(size=(n_s, 6)) * 1e-3, epj_disp=disp(n_j),
                   id_epj=np.arange(n_j, dtype=np.int32), spj_disp=disp(n_s), id_spj=np.arange(n_s, dtype=np.int32),
                   eps2=0.0, rcut2=0.02 ** 2, G=1.0)
    acc, pot, nnb = _run(wb)
    o = oracle.force(wb)
    assert (o["nnb"][::3] == n_j).all()
    assert_mixed_parity(acc, pot, nnb, o, f"r_search {rs}")


@pytest.mark.parametrize("n_pairs", [1, 16, 33, 200])
def test_companions_far_from_the_origin(n_pairs):
    rng = np.random.default_rng(n_pairs)
    nw, n_i, n_s, rs = 12, 2 * n_pairs, 30, 1e-5
    u = rng.normal(size=(nw * n_pairs, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    sep = rs * np.exp(rng.uniform(np.log(0.5), np.log(2.0), nw * n_pairs))
    sep[::4] = rs * (1 + rng.uniform(-1e-6, 1e-6, sep[::4].size))  # at the search radius, to a few roundings
    cen = np.array([3e4, -2e4, 1e4]) + np.repeat(rng.normal(size=(nw, 3)), n_pairs, axis=0)
    com = cen + rng.uniform(-0.05, 0.05, (nw * n_pairs, 3))
    pos = np.empty((nw * n_i, 3))
    pos[0::2], pos[1::2] = com + 0.5 * sep[:, None] * u, com - 0.5 * sep[:, None] * u
    ni = nw * n_i
    disp = np.arange(nw + 1, dtype=np.int64) * n_i
    wb = WalkBatch(epi_pos=pos, epi_rs=np.full(ni, rs), epi_disp=disp, epj_pos=pos, epj_mass=rng.uniform(0.1, 1, ni),
                   epj_rs=np.full(ni, rs), spj_pos=pos.mean(0) + rng.normal(size=(n_s, 3)) * 9,
                   spj_mass=rng.uniform(0.1, 1, n_s), spj_quad=np.zeros((n_s, 6)), epj_disp=disp,
                   id_epj=np.arange(ni, dtype=np.int32), spj_disp=np.arange(nw + 1, dtype=np.int64) * n_s,
                   id_spj=np.tile(np.arange(n_s, dtype=np.int32), nw), eps2=0.0, rcut2=1e-12, G=1.0)
    acc, pot, nnb = _run(wb)
    assert_mixed_parity(acc, pot, nnb, oracle.force(wb), f"{n_pairs} pairs")
