"""The work that users of this package have it do, through its public entry points.

Every case is one of the ways a star-cluster code reaches the soft force:

* ``call``: one multi-walk evaluation through the functor pair, host records
  in and host records out (EPJ/SPJ send, walk dispatch, retrieve), in one of
  the library's modes: soft force, plain FP64 soft force, fused changeover,
  neighbour search, KDKDK_4TH gradient pass;
* ``batches``: PeTar's unchanged call pattern, one send and then
  dispatch/retrieve pairs of 200 walks (its n_walk_limit);
* ``ensemble``: independent clusters joined in one launch, each walk with its
  cluster's cutoff;
* ``noalloc``: the allocation-free entry point on arrays in device memory;
* ``steps``: kick-drift-force-kick steps of the device-resident tree step,
  captured in a CUDA graph, and the new state read back.

The clusters are those of the package's configurations: Plummer spheres with a
Kroupa mass function, theta = 0.3 and up to half of the stars in binaries, and
King W0 = 7 models with theta = 0.4, from some hundred particles to
1,572,864, with the changeover radius shrinking as the cluster grows.

The mixed-precision kernels compute pairs and partial sums in FP32; the FP64
fields of the force records are their container.  Their accelerations and
potentials are returned as float32, the type they are computed in.  What is
computed in FP64 (the plain FP64 kernel, positions and velocities of the tree
step) is returned as float64, and neighbour counts as integers.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from petar_gb300 import gpuforce, ics, nbody, walks

WALKS_PER_CALL = 200  # PeTar's n_walk_limit
DT = 1.0 / 4096


def _r_out(n: int) -> float:
    """0.02 at 2,048 stars, 0.0070 at 65,536, 0.0031 at a million."""
    return 0.02 * (n / 2048.0) ** -0.3


def listed() -> list:
    return [
        # The headline workload: a million centres of mass, half of them binaries, one call for all walks.
        dict(name="call_1m_binaries", kind="call", mode="force", n=1048576, binaries=0.5, group=512),
        # A mid-size cluster without binaries, the commonest production size.
        dict(name="call_65k", kind="call", mode="force", n=65536, binaries=0.0, group=512),
        # A small open cluster: the call's latency, launches and copies.
        dict(name="call_700", kind="call", mode="force", n=700, binaries=0.0, group=512),
        # PeTar as it stands: 200 walks per functor call, 15 calls.
        dict(name="batches_262k_binaries", kind="batches", n=262144, binaries=0.5, group=512),
        # Independent clusters of odd sizes in one launch.
        dict(name="ensemble_12", kind="ensemble", clusters=12, n_min=1024, n_max=65536, binaries=0.3),
        # The FP64 option, for verification runs.
        dict(name="fp64_10k", kind="call", mode="fp64", n=10000, binaries=0.0, group=512),
        # The fused changeover correction of a binary-rich cluster.
        dict(name="changeover_131k_binaries", kind="call", mode="changeover", n=131072, binaries=0.5, group=512),
        # The second pass of the fourth-order integrator, in its default accuracy.
        dict(name="gradient_50k_binaries", kind="call", mode="gradient", n=50000, binaries=0.5, group=512),
        # Neighbour search alone.
        dict(name="search_200k_binaries", kind="call", mode="search", n=200000, binaries=0.5, group=512),
        # A code that owns its device memory, a cluster of odd size.
        dict(name="noalloc_33333", kind="noalloc", n=33333, binaries=0.0, group=512),
        # The device-resident step at a million stars, and where launches count.
        dict(name="steps_king_1m", kind="steps", n=1048576, steps=2, group=512),
        dict(name="steps_king_3k", kind="steps", n=3000, steps=2, group=512),
    ]


def draw(rng) -> dict:
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    group = rng.choice([256, 512, 512, 1024])
    binaries = rng.choice([0.0, 0.0, 0.3, 0.5])
    kind = rng.choice(["force", "force", "force", "fp64", "changeover", "gradient", "search", "batches", "ensemble",
                       "noalloc", "steps", "steps"])
    if kind == "force":
        return dict(kind="call", mode="force", n=size(500, 700000), binaries=binaries, group=group)
    if kind == "fp64":
        return dict(kind="call", mode="fp64", n=size(500, 20000), binaries=binaries, group=group)
    if kind in ("changeover", "gradient", "search"):
        return dict(kind="call", mode=kind, n=size(1000, 250000), binaries=binaries, group=group)
    if kind == "batches":
        return dict(kind="batches", n=size(20000, 400000), binaries=binaries, group=group)
    if kind == "ensemble":
        return dict(kind="ensemble", clusters=rng.randint(2, 20), n_min=1024, n_max=size(4000, 65536),
                    binaries=binaries)
    if kind == "noalloc":
        return dict(kind="noalloc", n=size(500, 200000), binaries=binaries, group=group)
    return dict(kind="steps", n=size(1000, 1000000), steps=rng.randint(1, 3), group=group)


# ---------------------------------------------------------------- inputs


def _cluster(case: dict, seed: int) -> ics.Cluster:
    if case["kind"] == "steps":
        cl = ics.make_king_cluster(seed, case["n"], _r_out(case["n"]), W0=7.0, theta=0.4)
        cl.n_group_limit = case["group"]
        return cl
    return ics.make_plummer_cluster(seed, case["n"], _r_out(case["n"]), binary_fraction=case["binaries"],
                                    n_group_limit=case["group"])


def _batch(case: dict, seed: int) -> walks.WalkBatch:
    if case["kind"] != "ensemble":
        return walks.build_walks(_cluster(case, seed))
    # Sizes spread evenly over the logarithm of the range; the seed makes the stars.
    n = np.exp(np.linspace(math.log(case["n_max"]), math.log(case["n_min"]), case["clusters"])).astype(int)
    return walks.concat_batches([
        walks.build_walks(ics.make_plummer_cluster(seed * 64 + k, int(m), 0.05 * float(m) ** (-1 / 3),
                                                   binary_fraction=case["binaries"])) for k, m in enumerate(n)])


def _changeover(case: dict, seed: int):
    """The batch with the changeover data of its stars (a tenth of them members, a twentieth artificial)."""
    wb = _batch(case, seed)
    r_out = _r_out(case["n"])
    return walks.make_changeover(wb, 0.1 * r_out, r_out, seed=seed)


def _accelerations(cl: ics.Cluster, wb: walks.WalkBatch) -> np.ndarray:
    """Accelerations for the gradient pass, as a first pass leaves them: the Plummer sphere's and, for the stars
    of binaries, the companion's with the linear cutoff."""
    r_scale = 3.0 * np.pi / 16.0
    acc = -cl.pos / ((cl.pos ** 2).sum(1) + r_scale ** 2)[:, None] ** 1.5
    n_bin = wb.meta["n_binary"]
    if n_bin:
        first = cl.n - 2 * n_bin
        p, m = cl.pos[first:], cl.mass[first:]
        d = p[1::2] - p[0::2]
        k = np.maximum((d * d).sum(1), cl.r_out ** 2) ** -1.5
        acc[first::2] += (m[1::2] * k)[:, None] * d
        acc[first + 1::2] -= (m[0::2] * k)[:, None] * d
    return np.ascontiguousarray(acc[wb.epi_index])


def _gradient(case: dict, seed: int):
    cl = _cluster(case, seed)
    wb = walks.build_walks(cl)
    wb.meta["n_binary"] = int(round(case["binaries"] * case["n"]))
    return wb, _accelerations(cl, wb)


_NOALLOC_EPJ = np.dtype([("pos", "<f8", 3), ("mass", "<f4"), ("r_search2", "<f4")])
_NOALLOC_SPJ = np.dtype([("pos", "<f8", 3), ("mass", "<f4"), ("pad0", "<f4"), ("quad_traceless", "<f4", 6),
                         ("trace", "<f4"), ("pad1", "<f4")])


def _noalloc_state(wb: walks.WalkBatch) -> dict:
    epj = np.zeros(wb.epj_mass.size, _NOALLOC_EPJ)
    epj["pos"], epj["mass"], epj["r_search2"] = wb.epj_pos, wb.epj_mass, wb.epj_rs * wb.epj_rs
    q = wb.spj_quad
    tr = q[:, 0] + q[:, 1] + q[:, 2]
    spj = np.zeros(wb.spj_mass.size, _NOALLOC_SPJ)
    spj["pos"], spj["mass"], spj["trace"] = wb.spj_pos, wb.spj_mass, tr
    spj["quad_traceless"] = 3.0 * q
    for d in range(3):
        spj["quad_traceless"][:, d] = 3.0 * q[:, d] - tr
    table = np.stack([wb.epi_disp[:-1], wb.n_epi, wb.epj_disp[:-1], wb.n_epj, wb.spj_disp[:-1], wb.n_spj],
                     axis=1).astype(np.int64)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()

    ni = wb.epi_rs.size
    f = gpuforce.load().pgf_force_device_noalloc
    vp, i64, cd = ctypes.c_void_p, ctypes.c_int64, ctypes.c_double
    f.argtypes = [ctypes.c_int, vp, vp, i64, vp, vp, i64, vp, i64, vp, i64, vp, i64, cd, cd, cd, vp, vp, vp,
                  ctypes.c_char_p, ctypes.c_size_t]
    f.restype = ctypes.c_int
    return dict(f=f, n_walk=wb.n_walk, table=dev(table),
                epi=dev(np.concatenate([wb.epi_pos, wb.epi_rs[:, None]], axis=1)), epj=dev(epj),
                epj_rs=dev(wb.epj_rs), spj=dev(spj), id_epj=dev(wb.id_epj), id_spj=dev(wb.id_spj),
                sizes=(ni, epj.size, spj.size, wb.id_epj.size, wb.id_spj.size), const=(wb.eps2, wb.rcut2, wb.G),
                accp=torch.zeros((ni, 4), dtype=torch.float64, device="cuda"),
                nnb=torch.zeros((ni,), dtype=torch.int32, device="cuda"), message=ctypes.create_string_buffer(256))


def _batch_slices(n_walk: int) -> list:
    return [(b, min(n_walk, b + WALKS_PER_CALL)) for b in range(0, n_walk, WALKS_PER_CALL)]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "steps":
        cl = _cluster(case, seed)
        h = nbody.DeviceNBody(cl)
        pin = dict(dtype=torch.float64, pin_memory=True)
        return dict(kind=kind, h=h, steps=case["steps"], pos=torch.empty((cl.n, 3), **pin),
                    vel=torch.empty((cl.n, 3), **pin), acc=torch.empty((cl.n, 3), **pin),
                    pot=torch.empty((cl.n,), **pin), nnb=torch.empty((cl.n,), dtype=torch.int32, pin_memory=True))
    if kind == "noalloc":
        return dict(kind=kind, **_noalloc_state(_batch(case, seed)))
    mode = case.get("mode", "force")
    if mode == "changeover":
        rec = gpuforce.Records(*_changeover(case, seed))
    elif mode == "gradient":
        wb, acc = _gradient(case, seed)
        rec = gpuforce.Records(wb, acc=(acc, acc))
    else:
        rec = gpuforce.Records(_batch(case, seed))
    n, words = rec.force.size, rec.force.dtype.itemsize // 8
    fields = torch.from_numpy(rec.force.view(np.float64).reshape(n, words))
    at = {k: v[1] // 8 for k, v in rec.force.dtype.fields.items()}
    return dict(kind=kind, mode=mode, rec=rec, fields=fields, at=at,
                accp=torch.empty((n, 4), dtype=torch.float32), extra=torch.empty((n, 3), dtype=torch.float32))


# ---------------------------------------------------------------- one pass


def _results(s: dict) -> dict:
    rec, at, f = s["rec"], s["at"], s["fields"]
    if s["mode"] == "search":
        return dict(n_ngb=rec.force["n_ngb"])
    out = dict(n_ngb=rec.force["n_ngb"])
    if s["mode"] == "fp64":
        out.update(acc=rec.force["acc"], pot=rec.force["pot"])
        return out
    # acc and pot lie side by side in the record
    s["accp"].copy_(f[:, at["acc"]:at["acc"] + 4])
    out["accp"] = s["accp"]
    if s["mode"] == "changeover":
        s["extra"][:, :1].copy_(f[:, at["pot_soft"]:at["pot_soft"] + 1])
        out["pot_soft"] = s["extra"][:, 0]
    if s["mode"] == "gradient":
        s["extra"].copy_(f[:, at["acorr"]:at["acorr"] + 3])
        out["acorr"] = s["extra"]
    return out


def _run_batches(s: dict) -> dict:
    rec = s["rec"]
    f = gpuforce.CalcForceWithLinearCutoffCUDAMultiWalk(0, rec.eps2, rec.rcut2, rec.G)
    f(0, 0, None, None, None, None, None, None, rec.epj, rec.epj.size, rec.spj, rec.spj.size, True)
    for a, b in _batch_slices(rec.n_walk):
        f(0, b - a, rec.p_epi[a:b], rec.n_epi[a:b], rec.p_id_epj[a:b], rec.n_epj[a:b], rec.p_id_spj[a:b],
          rec.n_spj[a:b], None, 0, None, 0, False, epi_dtype=rec.epi.dtype)
        gpuforce.RetrieveForceCUDA(0, b - a, rec.n_epi[a:b], rec.p_force[a:b], force_dtype=rec.force.dtype)
    return _results(s)


def _run_noalloc(s: dict) -> dict:
    ni, ne, ns, nie, nis = s["sizes"]
    rc = s["f"](s["n_walk"], s["table"].data_ptr(), s["epi"].data_ptr(), ni, s["epj"].data_ptr(),
                s["epj_rs"].data_ptr(), ne, s["spj"].data_ptr(), ns, s["id_epj"].data_ptr(), nie,
                s["id_spj"].data_ptr(), nis, *s["const"], s["accp"].data_ptr(), s["nnb"].data_ptr(),
                torch.cuda.current_stream().cuda_stream, s["message"], 256)
    if rc != 0:
        raise RuntimeError(s["message"].value.decode())
    return dict(accp=s["accp"].float(), n_ngb=s["nnb"])


def _run_steps(s: dict) -> dict:
    h = s["h"]
    h.run(s["steps"], DT)
    if gpuforce.load().pgf_nbody_get(h._h, s["pos"].data_ptr(), s["vel"].data_ptr(), s["acc"].data_ptr(),
                                     s["pot"].data_ptr(), s["nnb"].data_ptr()) != 0:
        raise RuntimeError("pgf_nbody_get")
    return dict(pos=s["pos"], vel=s["vel"], acc=s["acc"].float(), pot=s["pot"].float(), n_ngb=s["nnb"])


def run(s: dict) -> dict:
    if s["kind"] == "batches":
        return _run_batches(s)
    if s["kind"] == "noalloc":
        return _run_noalloc(s)
    if s["kind"] == "steps":
        return _run_steps(s)
    rec, mode = s["rec"], s["mode"]
    gpuforce.set_precision(gpuforce.PGF_PRECISION_FP64 if mode == "fp64" else gpuforce.PGF_PRECISION_MIXED)
    if mode == "changeover":
        gpuforce.set_changeover_layout(rec)
        gpuforce.set_mode(gpuforce.PGF_MODE_FORCE_CHANGEOVER)
    elif mode == "gradient":
        gpuforce.set_gradient_layout(rec)
        gpuforce.set_mode(gpuforce.PGF_MODE_GRADIENT)
    elif mode == "search":
        gpuforce.set_mode(gpuforce.PGF_MODE_NEIGHBOR_SEARCH)
    try:
        gpuforce.dispatch(rec)
        gpuforce.retrieve(rec)
    finally:
        gpuforce.set_precision(gpuforce.PGF_PRECISION_MIXED)
        gpuforce.set_mode(gpuforce.PGF_MODE_FORCE)
        if mode == "changeover":
            gpuforce.set_changeover_layout(None)
        elif mode == "gradient":
            gpuforce.set_gradient_layout(None)
    return _results(s)


# ---------------------------------------------------------------- work


def _estimate(n: int, binaries: float, group: int, theta: float = 0.3) -> tuple:
    """(particles, EP-EP pairs, EP-SP pairs) of one evaluation, from lists of seeded clusters of these
    models: lists grow with the logarithm of n and pairs with the group size."""
    full = int(round(n * (1 + binaries)))
    per_i_ep = min(full, 6300.0 * (0.3 / theta) ** 2.5 * (group / 512.0) ** 0.4)
    per_i_sp = min(0.25 * full, max(50.0, 1150.0 * (math.log2(max(full, 64)) - 12.6)) * (0.3 / theta) ** 2.2)
    return full, full * per_i_ep, full * per_i_sp


def work(case: dict) -> dict:
    kind, mode = case["kind"], case.get("mode", "force")
    if kind == "ensemble":
        lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
        n = [math.exp(lo + (hi - lo) * (k + 0.5) / case["clusters"]) for k in range(case["clusters"])]
        parts = [_estimate(int(m), case["binaries"], 512) for m in n]
        full, ep, sp = (sum(p[k] for p in parts) for k in range(3))
        group = 512
    else:
        group = case["group"]
        full, ep, sp = _estimate(case["n"], case.get("binaries", 0.0), group, 0.4 if kind == "steps" else 0.3)
    evaluations = case["steps"] if kind == "steps" else 1
    flops = ep * 19.0 + sp * 54.0
    if mode == "search":
        flops = ep * 9.0
    elif mode == "gradient":
        flops = ep * 45.0 + sp * 54.0
    # Lists (4 bytes an entry, one list for about 0.3 group particles), each record once in and out.
    entries = (ep + (0.0 if mode == "search" else sp)) / (0.29 * group)
    byts = full * (48.0 + 112.0 + 40.0) + 0.45 * full * 80.0 + (0.0 if kind == "steps" else 4.0 * entries)
    return {"bytes": evaluations * byts, "flops": evaluations * flops}


# ---------------------------------------------------------------- 64 bits, plain torch


def _dev(a) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda" if torch.cuda.is_available() else "cpu")


def _soft_force(wb: walks.WalkBatch, co=None, acc=None) -> dict:
    """The sums over the batch's lists in 64 bits: soft force with the linear cutoff and quadrupoles; with co the
    changeover correction of neighbours; with acc the gradient correction in the place of the EP-EP force."""
    xi_all, rs_all = _dev(wb.epi_pos), _dev(wb.epi_rs)
    xj_all, mj_all, rsj_all = _dev(wb.epj_pos), _dev(wb.epj_mass), _dev(wb.epj_rs)
    xs_all, ms_all, q_all = _dev(wb.spj_pos), _dev(wb.spj_mass), _dev(wb.spj_quad)
    ids_e, ids_s = _dev(wb.id_epj).long(), _dev(wb.id_spj).long()
    n = wb.epi_rs.size
    out = {k: torch.zeros((n, 3) if k in ("acc", "acorr") else n, dtype=torch.float64, device=xi_all.device)
           for k in ("acc", "pot", "pot_soft", "acorr")}
    if acc is not None:
        a_all = _dev(acc)
        out["acc"] += a_all
    if co is not None:
        ci = [_dev(a) for a in (co.epi_r_in, co.epi_r_out, co.epi_self_mass)]
        cj = [_dev(a) for a in (co.epj_r_in, co.epj_r_out, co.epj_mass_backup, co.epj_status)]
        idi, idj = _dev(co.epi_id), _dev(co.epj_id)
    for w in range(wb.n_walk):
        rc2 = float(wb.walk_rcut2[w]) if wb.walk_rcut2 is not None else wb.rcut2
        i0, i1 = int(wb.epi_disp[w]), int(wb.epi_disp[w + 1])
        je = ids_e[int(wb.epj_disp[w]):int(wb.epj_disp[w + 1])]
        js = ids_s[int(wb.spj_disp[w]):int(wb.spj_disp[w + 1])]
        rows = max(1, (1 << 25) // max(1, je.numel(), js.numel()))
        for b in range(i0, i1, rows):
            r = slice(b, min(i1, b + rows))
            xi = xi_all[r]
            d = [xj_all[je, c][None, :] - xi[:, c][:, None] for c in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + wb.eps2
            mj = mj_all[je][None, :]
            if acc is not None:
                da = [a_all[je, c][None, :] - a_all[r, c][:, None] for c in range(3)]
                r2m = r2.clamp_min(rc2)
                k = mj * r2m ** -1.5
                al = 3.0 * (d[0] * da[0] + d[1] * da[1] + d[2] * da[2]) / r2m
                for c in range(3):
                    out["acorr"][r, c] = 2.0 * (k * (da[c] - al * d[c])).sum(1)
            else:
                inv = r2.clamp_min(rc2).rsqrt()
                gm = mj * inv
                k = gm * inv * inv
                pot = -gm
                pot_soft = pot
                if co is not None:
                    near = (r2 < torch.maximum(rs_all[r][:, None], rsj_all[je][None, :]) ** 2) & \
                        (idi[r][:, None] != idj[je][None, :])
                    use_i = ci[1][r][:, None] > cj[1][je][None, :]
                    rin = torch.where(use_i, ci[0][r][:, None], cj[0][je][None, :])
                    rout = torch.where(use_i, ci[1][r][:, None], cj[1][je][None, :])
                    coff = (rout - rin) / (rout + rin)
                    dr = r2.sqrt()
                    x = (dr - rin) / (rout - rin)
                    xc = x.clamp(0.0, 1.0)
                    wacc = (xc - 1) ** 4 * (1 + 4 * xc + 10 * xc ** 2 + 20 * xc ** 3 + 35 * coff * xc ** 4)
                    wpot = torch.where(x >= 1, (1 + coff) / rout * dr,
                                       1 - coff * xc ** 5 * (5 * xc ** 3 - 20 * xc ** 2 + 28 * xc - 14))
                    mbk, status = cj[2][je][None, :], cj[3][je][None, :]
                    m_pot = torch.where((status == 0) & (mbk == 0), mj, torch.where(status < 0, mbk, 0.0 * mj))
                    k = torch.where(near, mj * (1 - wacc) / (r2 * dr), k)
                    pot = torch.where(near, -m_pot / dr, pot)
                    pot_soft = torch.where(near, -m_pot * (1 - wpot) / dr, pot_soft)
                for c in range(3):
                    out["acc"][r, c] = wb.G * (k * d[c]).sum(1)
                out["pot"][r] = wb.G * pot.sum(1)
                out["pot_soft"][r] = wb.G * pot_soft.sum(1)
                if co is not None:
                    self_term = wb.G * ci[2][r] / math.sqrt(rc2)
                    out["pot"][r] += self_term
                    out["pot_soft"][r] += self_term
            d = [xs_all[js, c][None, :] - xi[:, c][:, None] for c in range(3)]
            inv2 = 1.0 / (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + wb.eps2)
            inv = inv2.sqrt()
            q = [q_all[js, c][None, :] for c in range(6)]
            tr = q[0] + q[1] + q[2]
            qd = [q[0] * d[0] + q[3] * d[1] + q[4] * d[2], q[3] * d[0] + q[1] * d[1] + q[5] * d[2],
                  q[4] * d[0] + q[5] * d[1] + q[2] * d[2]]
            m, inv3 = ms_all[js][None, :], inv * inv2
            inv5 = 1.5 * inv3 * inv2
            qrr5 = (qd[0] * d[0] + qd[1] * d[1] + qd[2] * d[2]) * inv5
            k = m * inv3 - tr * inv5 + 5.0 * qrr5 * inv2
            pot = -wb.G * (m * inv - 0.5 * tr * inv3 + qrr5).sum(1)
            for c in range(3):
                out["acc"][r, c] += wb.G * (k * d[c] - 2.0 * inv5 * qd[c]).sum(1)
            out["pot"][r] += pot
            out["pot_soft"][r] += pot
    return out


def exact(case: dict, seed: int):
    kind, mode = case["kind"], case.get("mode", "force")
    if mode == "search":
        return None  # whole numbers only
    if kind == "steps":
        return _exact_steps(case, seed)
    if mode == "changeover":
        r = _soft_force(*_changeover(case, seed))
        return dict(accp=torch.cat([r["acc"], r["pot"][:, None]], 1), pot_soft=r["pot_soft"], n_ngb=None)
    if mode == "gradient":
        wb, acc = _gradient(case, seed)
        r = _soft_force(wb, acc=acc)
        return dict(accp=torch.cat([r["acc"], r["pot"][:, None]], 1), acorr=r["acorr"], n_ngb=None)
    r = _soft_force(_batch(case, seed))
    if mode == "fp64":
        return dict(acc=r["acc"], pot=r["pot"], n_ngb=None)
    return dict(accp=torch.cat([r["acc"], r["pot"][:, None]], 1), n_ngb=None)


def _exact_steps(case: dict, seed: int) -> dict:
    """The same steps with 64-bit forces.  The lists at each step's positions are inputs here: those of the host
    list builder."""
    cl = _cluster(case, seed)

    def force():
        wb = walks.build_walks(cl)
        r = _soft_force(wb)
        acc, pot = np.empty((cl.n, 3)), np.empty(cl.n)
        acc[wb.epi_index], pot[wb.epi_index] = r["acc"].cpu().numpy(), r["pot"].cpu().numpy()
        return acc, pot

    acc, pot = force()
    for _ in range(case["steps"]):
        cl.vel = cl.vel + 0.5 * DT * acc
        cl.pos = cl.pos + DT * cl.vel
        acc, pot = force()
        cl.vel = cl.vel + 0.5 * DT * acc
    return dict(pos=cl.pos, vel=cl.vel, acc=acc, pot=pot, n_ngb=None)
