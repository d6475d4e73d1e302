"""Performance cases of the per-iteration hot path: what a user's program asks of the library.

A pass of most cases is what a driver program does with the solver it keeps: hand over the state
in its page-locked host arrays, advance it, and take the state back.  The solver (its grid,
geometry, work lists and tuned sweep schedule) is prepared once, as a program keeps it over a run.
Two cases are single stages with a closed 64-bit value: the spectral radius and gradient
subroutines, and the block metrics with the wall distance.

Grids, schemes and precisions are those of the repository's configurations (channel bump,
five-block cascade and its serving levels, annular sector, square cylinder), at sizes from the
smallest test block to the benchmark cascade.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from trans_gb300 import abi
from trans_gb300 import case as CS
from trans_gb300 import cases
from trans_gb300 import native
from trans_gb300.solver import Batch, Solver, block_metrics_gpu, device_block_metrics

UP = ("V", "PP", "T", "RMIU", "WT0", "WT1")       # what a time-marching program hands over
DOWN = ("V", "PP", "T", "RMIU")                   # and takes back
G = 2                                             # array offset of index 0 (arrays start at -2)


def listed():
    return [
        # the smallest test block, MDCD + AUSMPW+: launch and dependency latency alone
        dict(name="channel_tiny_fp64", kind="march", grid="channel", ni=25, nj=17, nk=6, precision="fp64",
             spatial=3, roe=3, iters=20),
        # the channel bump at its stated size 97x49x9, MUSCL + Roe (the plain FP64 method)
        dict(name="channel_fp64", kind="march", grid="channel", ni=97, nj=49, nk=9, precision="fp64",
             spatial=2, roe=1, iters=20),
        # the same block in mixed precision: an ordinary small interactive solve
        dict(name="channel_mixed", kind="march", grid="channel", ni=97, nj=49, nk=9, precision="mixed",
             spatial=2, roe=1, iters=20),
        # rotating annular sector, Runge-Kutta stages, odd sizes (rotor-frame explicit marching)
        dict(name="annulus_rk3_fp64", kind="march", grid="annulus", ni=71, nj=39, nk=27, precision="fp64",
             spatial=3, roe=1, rk=1, iters=4),
        # the serving stream's most frequent request: coarse cascade, both precisions
        dict(name="cascade_coarse_fp64", kind="march", grid="cascade", ns=60, npitch=16, nte=4, nr=48, nh=32, nk=32,
             precision="fp64", spatial=3, roe=3, iters=6),
        dict(name="cascade_coarse_mixed", kind="march", grid="cascade", ns=60, npitch=16, nte=4, nr=48, nh=32, nk=32,
             precision="mixed", spatial=2, roe=1, iters=16),
        # the benchmark cascade, 1,966,080 cells: the headline FP64 path and the mixed path
        dict(name="cascade_full_fp64", kind="march", grid="cascade", ns=96, npitch=32, nte=16, nr=48, nh=64, nk=64,
             precision="fp64", spatial=3, roe=3, iters=3),
        dict(name="cascade_full_mixed", kind="march", grid="cascade", ns=96, npitch=32, nte=16, nr=48, nh=64, nk=64,
             precision="mixed", spatial=3, roe=3, iters=16),
        # one physical step (10 dual-time sub-iterations) of the square-cylinder DES
        dict(name="cylinder_des_mixed", kind="march", grid="cylinder", ni=193, nj=97, nk=49, precision="mixed",
             spatial=3, roe=3, iters=2),
        # requests of uneven size resident together, as the serving loop holds them
        dict(name="batch_mixed", kind="batch", coarse=4, medium=1, precision="mixed", spatial=3, roe=3, iters=8),
        # the spectral radius and gradient subroutines as single drop-ins
        dict(name="stages_fp64", kind="stages", grid="annulus", ni=129, nj=65, nk=49, precision="fp64", spatial=2, roe=1),
        # set-up of a request: block metrics and wall distance of the coarse cascade's O-block
        dict(name="geometry_oblock", kind="geometry", ns=60, npitch=16, nte=4, nr=48, nh=32, nk=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_cascade(rng, most):
    """Cascade sizes (odd ones among them) up to `most` times the coarse level's extents."""
    nte = rng.choice((2, 4, 8))
    return dict(ns=_log_int(rng, 20, int(60 * most)), npitch=rng.randint(8, 28), nte=nte, nr=rng.randint(12, 48),
                nh=_log_int(rng, 10, int(32 * most)), nk=2 * _log_int(rng, 6, int(16 * most)))


def draw(rng):
    kind = rng.choice(("march", "march", "march", "march", "batch", "stages", "geometry"))
    if kind == "batch":
        return dict(kind="batch", coarse=rng.randint(1, 5), medium=rng.randint(0, 1), precision="mixed", spatial=rng.choice((2, 3)),
                    roe=3, iters=rng.randint(3, 10))
    if kind == "stages":
        return dict(kind="stages", grid="annulus", ni=_log_int(rng, 17, 161), nj=_log_int(rng, 11, 65), nk=_log_int(rng, 7, 49),
                    precision="fp64", spatial=2, roe=1)
    if kind == "geometry":
        return dict(kind="geometry", **_draw_cascade(rng, 1.0))
    precision = rng.choice(("fp64", "mixed"))
    spatial, roe = rng.choice(((2, 1), (2, 3), (3, 1), (3, 3)))
    scheme = dict(precision=precision, spatial=spatial, roe=roe)
    grid = rng.choice(("channel", "cascade", "cascade", "annulus", "cylinder"))
    if grid == "channel":
        return dict(kind="march", grid=grid, ni=_log_int(rng, 17, 161), nj=_log_int(rng, 13, 97), nk=_log_int(rng, 5, 33),
                    iters=rng.randint(2, 12), **scheme)
    if grid == "annulus":
        return dict(kind="march", grid=grid, ni=_log_int(rng, 17, 129), nj=_log_int(rng, 11, 65), nk=_log_int(rng, 7, 49),
                    rk=rng.randint(0, 1), iters=rng.randint(2, 5), **scheme)
    if grid == "cylinder":
        return dict(kind="march", grid=grid, ni=4 * _log_int(rng, 12, 48) + 1, nj=_log_int(rng, 25, 97), nk=_log_int(rng, 9, 49),
                    precision="mixed", spatial=3, roe=3, iters=1)
    return dict(kind="march", grid=grid, iters=rng.randint(2, 4), **_draw_cascade(rng, 1.4), **scheme)


# ------------------------------------------------------------------------------------------
# what a program has in hand before it iterates
# ------------------------------------------------------------------------------------------
def _grid_key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "kind", "iters")))


def _make(d):
    prec = abi.TRANS_MIXED if d["precision"] == "mixed" else abi.TRANS_FP64
    sw = dict(precision=prec, Kind_Spatial=d["spatial"], Kind_Roe=d["roe"])
    if d.get("rk"):
        sw.update(IF_RK=1, CFL_Sub_start=1.0, CFL_Sub_end=1.0)
    g = d["grid"]
    if g == "channel":
        return cases.channel_bump(ni=d["ni"], nj=d["nj"], nk=d["nk"], **sw)
    if g == "annulus":
        return cases.annular_sector(ni=d["ni"], nj=d["nj"], nk=d["nk"], rpm=2000.0, casing_kindsub=1, **sw)
    if g == "cylinder":
        return cases.square_cylinder(ni=d["ni"], nj=d["nj"], nk=d["nk"], perturbation=0.0, **sw)
    return cases.cascade(ns=d["ns"], npitch=d["npitch"], nle=2 * d["nte"], nte=d["nte"], nr=d["nr"], nh=d["nh"], nk=d["nk"], **sw)


@functools.lru_cache(maxsize=24)
def _set_up(key):
    """Case, connectivity, geometry and unperturbed initial field of a grid (no seed in them)."""
    c = _make(dict(key))
    conns, geo = CS.compute_geometry(c, metrics_fn=device_block_metrics())
    return c, conns, geo, CS.initial_state(c, geo, Q_dst=c.meta["Q_dst"], noise=0.0)


def _state(c, base, seed):
    """The initial field with a seeded perturbation: 1e-4 on the density, and 1% on the streamwise
    velocity where the configuration asks for one (the cylinder's wake)."""
    rng = np.random.default_rng(seed)
    p, out = c.params, {}
    for b in c.blocks:
        ni, nj, nk = b.dims
        i = (slice(G + 1, G + ni), slice(G + 1, G + nj), slice(G + 1, G + nk))
        s = {f: base[b.id][f].copy(order="F") for f in ("V", "PP", "T", "RMIU")}
        V = s["V"]
        V[(0,) + i] *= 1.0 + 1.0e-4 * rng.standard_normal(V[(0,) + i].shape)
        if c.name.startswith("square_cylinder"):
            e = 0.5 * V[(1,) + i] ** 2
            V[(1,) + i] *= 1.0 + 0.01 * rng.standard_normal(e.shape)
            V[(4,) + i] += 0.5 * V[(1,) + i] ** 2 - e
        s["T"][i] = p.RXM2 * s["PP"][i] / V[(0,) + i]
        s["WT0"], s["WT1"] = V, V
        out[b.id] = s
    return out


def _pinned(arr):
    """A page-locked Fortran-order copy of an array, as the caller's buffers are."""
    t = torch.empty(max(arr.size, 1), dtype=torch.float64, pin_memory=True)
    a = t.numpy()[:arr.size].reshape(arr.shape, order="F")
    a[...] = arr
    return a, t


class _Table:
    """The (block, field, array) lists of trans_set_fields / trans_get_fields."""

    def __init__(self, items):
        n = len(items)
        self.n, self.items = n, items
        self.ib, self.fid, self.ptr = (C.c_int * n)(), (C.c_int * n)(), (C.POINTER(C.c_double) * n)()
        for q, (ib, f, a, _) in enumerate(items):
            self.ib[q], self.fid[q], self.ptr[q] = ib, abi.FIELD_ID[f], a.ctypes.data_as(C.POINTER(C.c_double))

    def args(self):
        return self.n, self.ib, self.fid, self.ptr


def _up_table(c, st, fields=UP):
    return _Table([(ib, f, *_pinned(CS.fortran_view(f, st[b.id][f]))) for ib, b in enumerate(c.blocks) for f in fields])


def _down_table(c, fields=DOWN):
    return _Table([(ib, f, *_pinned(np.zeros(abi.field_shape(f, *b.dims), order="F"))) for ib, b in enumerate(c.blocks) for f in fields])


def _ok(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} failed ({rc})")


def _batch_members(case):
    lv = [dict(ns=60, npitch=16, nte=4, nr=48, nh=32, nk=32)] * case["coarse"] + [dict(ns=120, npitch=16, nte=4, nr=48, nh=64, nk=64)] * case["medium"]
    return [dict(grid="cascade", precision=case["precision"], spatial=case["spatial"], roe=case["roe"], **g) for g in lv]


def prepare(case, seed):
    lib = native.load()
    if case["kind"] == "geometry":
        d = dict(case, grid="cascade", precision="fp64", spatial=3, roe=3)
        c = _make({k: v for k, v in d.items() if k not in ("name", "kind")})
        rng = np.random.default_rng(seed)
        # another design each time: the grid stretched by up to 5% along each axis
        f = 1.0 + 0.05 * rng.random(3)
        c.blocks[0].xyz = c.blocks[0].xyz * f
        return dict(case=case, lib=lib, block=c.blocks[0], surfaces=[s * f for s in c.surfaces], tiny=c.params.Tiny)
    if case["kind"] == "batch":
        bt = Batch(abi.TRANS_MIXED if case["precision"] == "mixed" else abi.TRANS_FP64)
        ids, ups, downs = [], [], []
        for q, d in enumerate(_batch_members(case)):
            c, conns, geo, base = _set_up(_grid_key(d))
            st = _state(c, base, 1000 * seed + q)
            ids.append(bt.add(c, conns, geo, st))
            ups.append(_up_table(c, st))
            downs.append(_down_table(c, ("V",)))
        _ok(lib.trans_prepare(bt.ctx, 1), "trans_prepare")
        return dict(case=case, lib=lib, batch=bt, ids=ids, ups=ups, downs=downs)
    c, conns, geo, base = _set_up(_grid_key(case))
    st = _state(c, base, seed)
    s = Solver(c, conns, geo, st, lib)
    if case["kind"] == "stages":
        # the state with its ghost layers, as a program holds it after the boundary subroutine
        s.run_stage("BC_STATE", 1)
        st = {b.id: {f: s.get_field(ib, f) for f in DOWN} for ib, b in enumerate(c.blocks)}
        return dict(case=case, lib=lib, solver=s, up=_up_table(c, st, DOWN), down=_down_table(c, ("RDS", "DTM", "DQDXYZ", "SHOCK")), geo=geo, st=st)
    _ok(lib.trans_prepare(s.ctx, 1), "trans_prepare")
    return dict(case=case, lib=lib, solver=s, up=_up_table(c, st), down=_down_table(c))


def run(state):
    case, lib = state["case"], state["lib"]
    if case["kind"] == "geometry":
        return block_metrics_gpu(lib, state["block"], state["surfaces"], state["tiny"])
    if case["kind"] == "batch":
        bt = state["batch"]
        for cid, up in zip(state["ids"], state["ups"]):
            _ok(lib.trans_batch_set_fields(bt.ctx, cid, *up.args()), "trans_batch_set_fields")
        if bt.iterate(case["iters"]):
            raise RuntimeError("NaN")
        for cid, down in zip(state["ids"], state["downs"]):
            _ok(lib.trans_batch_get_fields(bt.ctx, cid, *down.args()), "trans_batch_get_fields")
        return {"case%d" % q: [a for _, _, a, _ in down.items] for q, down in enumerate(state["downs"])}
    s, up, down = state["solver"], state["up"], state["down"]
    _ok(lib.trans_set_fields(s.ctx, *up.args()), "trans_set_fields")
    out = {}
    if case["kind"] == "stages":
        s.run_stage("SPECRAD", 1)
        s.run_stage("GRADIENT", 1)
    else:
        for ki in range(1, case["iters"] + 1):
            norms = s.iterate(ki)
        out["residual"] = np.array([[n["DRSa"], n["DUa"], n["DRSk"], n["DRSo"]] for n in norms])
    _ok(lib.trans_get_fields(s.ctx, *down.args()), "trans_get_fields")
    for ib, f, a, _ in down.items:
        out["%s%d" % (f, ib)] = a
    return out


def _cells(case):
    """Interior cells, and cells with ghosts, of what the case iterates."""
    def blocks(d):
        g = d["grid"]
        if g != "cascade":
            return [(d["ni"], d["nj"], d["nk"])]
        nle, nk = 2 * d["nte"], d["nk"] + 1
        h = (d["nh"] + 1, 2 * d["npitch"] + nle + 1, nk)
        p = (d["ns"] + 1, d["npitch"] + 1, nk)
        return [(2 * d["nte"] + 2 * d["ns"] + nle + 1, d["nr"] + 1, nk), h, h, p, p]
    if case["kind"] == "batch":
        every = [b for d in _batch_members(case) for b in blocks(d)]
    elif case["kind"] == "geometry":
        every = blocks(dict(case, grid="cascade"))[:1]
    else:
        every = blocks(case)
    return sum((a - 1) * (b - 1) * (c - 1) for a, b, c in every), sum((a + 5) * (b + 5) * (c + 5) for a, b, c in every)


def work(case):
    n, padded = _cells(case)
    if case["kind"] == "geometry":
        # nodes in, 24 metric arrays out; every cell meets every wall panel (8 operations a pair)
        loop = 4 * case["nte"] + 2 * case["ns"]
        face = (case["nh"] * (2 * case["npitch"] + 2 * case["nte"]) + case["ns"] * case["npitch"]) * 2 + loop * case["nr"]
        panels = loop * case["nk"] + 2 * face
        return {"bytes": 8.0 * (3 * n + 24 * padded + 12 * panels), "flops": 8.0 * n * panels + 250.0 * n}
    if case["kind"] == "stages":
        # state 10 and metrics 17 words in, 3 + 1 + 18 + 1 out, once over the link and once on the card
        return {"bytes": 8.0 * (10 * padded + 17 * n + 23 * n), "flops": 420.0 * n}
    steps = case["iters"] * (10 if case.get("grid") == "cylinder" else 3 if case.get("rk") else 1)
    # per cell-iteration: state 10, two older time levels 14 and metrics 19 words in, state 10 and the
    # time levels 14 out; around a pass the state goes up (24 words) and comes back (10, a batch 7)
    down = 7 if case["kind"] == "batch" else 10
    return {"bytes": 8.0 * (67 * n * steps + (24 + down) * padded), "flops": 6000.0 * n * steps}


# ------------------------------------------------------------------------------------------
# the single stages in 64 bits, without the library
# ------------------------------------------------------------------------------------------
def _exact_stages(case, seed):
    s = prepare(case, seed)
    p = s["solver"].params
    out = {}
    for ib, b in enumerate(s["solver"].blocks):
        ni, nj, nk = b.dims
        st, g = s["st"][b.id], s["geo"][b.id]
        V, PP, T, mut = st["V"], st["PP"], st["T"], st["RMIU"]
        i = (slice(G + 1, G + ni), slice(G + 1, G + nj), slice(G + 1, G + nk))

        def at(a, d, o):        # the cells shifted by o along direction d
            q = list(i)
            q[d] = slice(i[d].start + o, i[d].stop + o)
            return a[tuple(q)]
        with np.errstate(all="ignore"):
            prim = [V[1] / V[0], V[2] / V[0], V[3] / V[0], T, V[5] / V[0], V[6] / V[0]]
            SD, AL, vol = g["SD"], g["ALAGM"], g["VOL"][i]
            # TIME_SpectralRadius
            rho, TT, m = V[0][i], T[i], mut[i]
            tc = TT * p.Csth1
            mu = (1.0 + p.Csthlnd) / (tc + p.Csthlnd) * tc ** 1.5
            visc = np.maximum((mu + m + 1e-20) * 4.0 / 3.0, (mu / 0.72 + m / 0.9 + 1e-20) * 1.4) / rho
            snd = np.sqrt(1.4 * PP[i] / rho)
            rd = []
            for d in range(3):
                A = [0.5 * (SD[d, k][i] + at(SD[d, k], d, 1)) for k in range(3)]
                s2 = A[0] ** 2 + A[1] ** 2 + A[2] ** 2
                rd.append(np.abs(sum(prim[k][i] * A[k] for k in range(3))) + np.sqrt(s2) * snd + 2.0 * s2 / vol * visc / p.Ref)
            dtm = p.CFL_Sub_end * vol / (rd[0] + rd[1] + rd[2]) if p.IF_Local_Sub == 1 else np.full(vol.shape, p.DT_LUSGS_Sub)
            # Green-Gauss gradients from length-weighted face averages
            grad = np.zeros((18,) + vol.shape)
            for q, f in enumerate(prim):
                for d in range(3):
                    al = AL[d]
                    fw = (al[i] * at(f, d, -1) + at(al, d, -1) * f[i]) / (al[i] + at(al, d, -1))
                    fe = (at(al, d, 1) * f[i] + al[i] * at(f, d, 1)) / (at(al, d, 1) + al[i])
                    for k in range(3):
                        grad[3 * q + k] += (fe * at(SD[d, k], d, 1) - fw * SD[d, k][i]) / vol
            u, v, w = grad[0:3], grad[3:6], grad[6:9]
            vort2 = (u[1] - v[0]) ** 2 + (u[2] - w[0]) ** 2 + (v[2] - w[1]) ** 2
            div2 = u[0] ** 2 + v[1] ** 2 + w[2] ** 2
            sens = div2 / np.maximum(div2 + vort2, 1.0)

        def laid_out(name, val, lead=()):
            a = np.zeros(lead + (ni + 5, nj + 5, nk + 5))
            a[(Ellipsis,) + i] = val
            o = abi.FIELD_LAYOUT[name][1] + G
            return a[(slice(None),) * len(lead) + (slice(o, None),) * 3]
        sh = np.zeros((ni + 5, nj + 5, nk + 5))
        sh[i] = sens
        for L in (1, 2, 3):     # the three ghost layers of a face take the adjacent cell's value
            for lo, hi, put in ((G + 1, G + 1 - L, 0), (G + ni - 1, G + ni - 1 + L, 0), (G + 1, G + 1 - L, 1),
                                (G + nj - 1, G + nj - 1 + L, 1), (G + 1, G + 1 - L, 2), (G + nk - 1, G + nk - 1 + L, 2)):
                src, dst = list(i), list(i)
                src[put], dst[put] = lo, hi
                sh[tuple(dst)] = sh[tuple(src)]
        out["RDS%d" % ib] = laid_out("RDS", np.stack(rd), (3,))
        out["DTM%d" % ib] = laid_out("DTM", dtm)
        out["DQDXYZ%d" % ib] = laid_out("DQDXYZ", grad, (18,))
        out["SHOCK%d" % ib] = sh
    return out


def _exact_geometry(case, seed):
    s = prepare(case, seed)
    X = s["block"].xyz
    ni, nj, nk = (n - 1 for n in X.shape[:3])
    full = (ni + 6, nj + 6, nk + 6)
    i = (slice(G + 1, G + 1 + ni), slice(G + 1, G + 1 + nj), slice(G + 1, G + 1 + nk))

    def corner(a, b, c):
        return X[a:ni + a, b:nj + b, c:nk + c]
    cen = sum(corner(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)) / 8.0
    out = {n: np.zeros(full) for n in ("XC", "YC", "ZC", "DST", "VOL", "RAD", "THTC", "ALENG", "ASENG")}
    SD, GR, AL = np.zeros((3, 3) + full), np.zeros((3,) + full), np.zeros((3,) + full)
    # distance to the nearest wall panel centre
    pan = np.concatenate([((S[:-1, :-1] + S[1:, :-1] + S[:-1, 1:] + S[1:, 1:]) / 4.0).reshape(-1, 3) for S in s["surfaces"]])
    pts = torch.from_numpy(np.ascontiguousarray(cen.reshape(-1, 3))).cuda()
    pan = torch.from_numpy(np.ascontiguousarray(pan)).cuda()
    dst = torch.empty(len(pts), dtype=torch.float64, device="cuda")
    for k in range(0, len(pts), 4096):
        d = pts[k:k + 4096, None, 0] - pan[None, :, 0]
        r = d * d
        for q in (1, 2):
            d = pts[k:k + 4096, None, q] - pan[None, :, q]
            r += d * d
        dst[k:k + 4096] = r.amin(1)
    out["DST"][i] = np.sqrt(np.maximum(dst.cpu().numpy(), s["tiny"])).reshape(ni, nj, nk)
    out["RAD"][i] = np.hypot(cen[..., 1], cen[..., 2])
    out["THTC"][i] = np.arctan2(cen[..., 2], cen[..., 1])
    # face vectors: half the cross product of the face diagonals, oriented along +d
    vol = np.zeros((ni, nj, nk))
    fcen = []
    for d in range(3):
        Y = np.moveaxis(X, d, 0)                        # node planes normal to d
        a, b = Y[:, 1:, 1:] - Y[:, :-1, :-1], Y[:, :-1, 1:] - Y[:, 1:, :-1]
        n = 0.5 * np.cross(a, b)
        mid = (Y[:, :-1, :-1] + Y[:, 1:, :-1] + Y[:, :-1, 1:] + Y[:, 1:, 1:]) / 4.0
        sgn = np.sign(np.sum(n[0] * (mid[1] - mid[0])))
        n = np.moveaxis(n * sgn, 0, d)
        area = np.sqrt(np.sum(n * n, -1) + s["tiny"])
        j = list(i)
        j[d] = slice(G + 1, G + 2 + (ni, nj, nk)[d])
        for k in range(3):
            SD[(d, k) + tuple(j)] = n[..., k]
        GR[(d,) + tuple(j)] = area
        lo, first = list(j), list(j)
        lo[d], first[d] = G, G + 1
        for k in range(3):
            SD[(d, k) + tuple(lo)] = SD[(d, k) + tuple(first)]
        GR[(d,) + tuple(lo)] = GR[(d,) + tuple(first)]
        AL[(d,) + i] = np.moveaxis(np.sqrt(np.sum((mid[1:] - mid[:-1]) ** 2, -1)), 0, d)
        fcen.append(mid)
        diag = corner(1, 1, 1) - corner(*[0 if q == d else 1 for q in range(3)])
        lower = tuple(slice(0, m) for m in (ni, nj, nk))
        vol += np.sum(diag * n[lower], -1) / 3.0
    out["VOL"][i] = vol
    # cell centres with the boundary face centres in the first ghost layer, then the distances to
    # the six neighbours (a direction of two cells left out)
    XYZ = np.zeros(full + (3,))
    XYZ[i] = cen
    for d in range(3):
        for at, plane in ((G, 0), (G + 1 + (ni, nj, nk)[d], -1)):
            j = list(i)
            j[d] = at
            XYZ[tuple(j)] = fcen[d][plane]
    far = []
    for d in range(3):
        for o in (-1, 1):
            j = list(i)
            j[d] = slice(i[d].start + o, i[d].stop + o)
            far.append((d, np.sqrt(np.sum((XYZ[tuple(j)] - cen) ** 2, -1))))
    least = [d for d in range(3) if (ni, nj, nk)[d] == 2]
    use = [v for d, v in far if not least or d != least[-1]]
    out["ALENG"][i], out["ASENG"][i] = np.maximum.reduce(use), np.minimum.reduce(use)
    out["XC"], out["YC"], out["ZC"] = XYZ[..., 0], XYZ[..., 1], XYZ[..., 2]
    out["SD"], out["GRAD"], out["ALAGM"] = SD, GR, AL
    return out


def exact(case, seed):
    """The two single stages.  A march has no value here: several iterations of the whole coupled
    path (boundaries, reconstruction, fluxes, ordered Gauss-Seidel sweeps, limited updates) take
    numpy minutes, as every hyperplane of every sweep is a step of its own."""
    if case["kind"] == "stages":
        return _exact_stages(case, seed)
    if case["kind"] == "geometry":
        return _exact_geometry(case, seed)
    return None
