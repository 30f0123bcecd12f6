"""Performance cases of the SN transport solve, through the calls that a user's program makes.

A case is a dict of plain values; `kind` says which entry point it goes through:

- "slab" / "grid": one 1D or one 2D/3D solve. entry "dropin" is compute_flux_tables (upload,
  solve, download, release on the default context: what replaces compute_flux(::SN)); entry
  "resident" solves a problem that stays uploaded (Context.solve + Context.download: the program
  that re-solves a plan it keeps).
- "batch": many resident slabs in one Context.solve_batch, every result downloaded.
- "serving": a burst of requests through ServingLoop (rb_submit / rb_poll).
- "coupled": transport_tables, the generation loop over photon, electron and positron.

Cross sections are the synthetic tables of radiant_b200.workloads (seeded); geometries, angular
orders and closures are those of the slab, grid and serving configurations there and of the
tests, over their sizes. `exact` is a plain torch solver in 64 bits of the same equations.
"""
import math
import os
import sys
import weakref

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "radiant.jl_b200"))

from radiant_b200 import serving as SV  # noqa: E402
from radiant_b200 import sn_flux as SN  # noqa: E402
from radiant_b200 import sources as SRC  # noqa: E402
from radiant_b200 import transport as TR  # noqa: E402
from radiant_b200 import workloads as W  # noqa: E402
from radiant_b200._abi import PackedProblem, ResultBuffers  # noqa: E402


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a short photon slab, everything on the host before and after
        _slab("slab-small", 53, 10, 8, 3),
        # the 1D photon slab configuration (200 voxels, S16, P7, 40 groups) as the drop-in call
        _slab("slab-photon", 200, 40, 16, 7, tol=1e-8),
        # the 1D electron slab configuration (linear DG in x and E, Fokker-Planck, S32, P15)
        _slab("slab-electron-dg", 300, 40, 32, 15, particle="electron", order=2, tol=1e-8, entry="resident"),
        # a treatment-planning style batch of ragged slabs in one launch, both arithmetic forms
        {"name": "batch-fp64", "kind": "batch", "count": 24, "max_cells": 700, "max_groups": 40, "precision": "fp64",
         "mix": 11},
        {"name": "batch-mixed", "kind": "batch", "count": 60, "max_cells": 500, "max_groups": 24, "precision": "mixed",
         "mix": 12},
        # the 2D photon configuration's shape (128 x 128, S12, Galerkin basis), few groups
        _grid("grid2d-photon", (128, 128), 2, 12, 5, accel="gmres", tol=1e-7),
        # ragged 2D electrons (CSD + Fokker-Planck) in the mixed form
        _grid("grid2d-electron-mixed", (97, 61), 4, 8, 5, particle="electron", accel="gmres", tol=1e-7, precision="mixed"),
        # 2D linear DG cells (full coupling, four moments per cell), odd sizes, as the drop-in call
        _grid("grid2d-dg", (41, 30), 2, 6, 3, order=2, accel="gmres", tol=1e-7, entry="dropin"),
        # the 3D photon configuration (64 cubed, S8, reflective Z-, BiCGStab) in the mixed form
        _grid("grid3d-photon-mixed", (64, 64, 64), 2, 8, 3, accel="bicgstab", tol=1e-6, precision="mixed", bcz=1),
        # ragged 3D electrons, plain FP64
        _grid("grid3d-electron", (48, 41, 35), 2, 8, 3, particle="electron", accel="bicgstab", tol=1e-6),
        # a burst of serving requests: 1D and 2D, photon or photon + electron + positron sets
        {"name": "serving", "kind": "serving", "count": 12, "max_cells": 600, "max_groups": 30, "max_side": 64,
         "precision": "mixed", "mix": 13},
        # coupled photon-electron-positron transport of a slab
        {"name": "coupled-slab", "kind": "coupled", "cells": 60, "groups": 10, "sn": 8, "legendre": 3},
    ]


def _slab(name, cells, groups, sn, legendre, particle="photon", order=1, tol=1e-7, precision="fp64", accel="gmres",
          entry="dropin"):
    return {"name": name, "kind": "slab", "cells": cells, "groups": groups, "sn": sn, "legendre": legendre,
            "particle": particle, "order": order, "tol": tol, "precision": precision, "accel": accel, "entry": entry}


def _grid(name, ns, groups, sn, legendre, particle="photon", order=1, tol=1e-7, precision="fp64", accel="gmres",
          entry="resident", bcz=0):
    return {"name": name, "kind": "grid", "nx": ns[0], "ny": ns[1], "nz": ns[2] if len(ns) > 2 else 0,
            "groups": groups, "sn": sn, "legendre": legendre, "particle": particle, "order": order, "tol": tol,
            "precision": precision, "accel": accel, "entry": entry, "bcz": bcz}


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["slab", "slab", "batch", "grid2", "grid2", "grid3", "grid3", "dg2", "serving"])
    particle = rng.choice(["photon", "electron"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "slab":
        order = rng.choice([1, 2])
        c = _slab("", log(50, 600), log(8, 60), rng.choice([8, 16, 32]), rng.randint(3, 7), particle, order,
                  precision=precision, accel=rng.choice(["gmres", "gmres", "bicgstab", "anderson", "livolant"]),
                  entry=rng.choice(["dropin", "resident"]))
    elif kind == "batch":
        c = {"kind": "batch", "count": rng.randint(6, 64), "max_cells": log(100, 600), "max_groups": rng.randint(12, 30),
             "precision": precision, "mix": rng.randint(0, 10 ** 6)}
    elif kind == "grid2":
        sn = rng.choice([4, 6, 8, 10, 12])
        side = 128 if sn <= 8 else 110
        c = _grid("", (log(24, side), log(24, side)), rng.randint(1, 3), sn, rng.randint(1, 5), particle,
                  precision=precision, accel=rng.choice(["gmres", "bicgstab"]), entry=rng.choice(["dropin", "resident"]))
    elif kind == "grid3":
        sn = rng.choice([4, 6, 8])
        c = _grid("", (log(15, 56), log(15, 56), log(15, 56)), rng.randint(1, 2), sn, 3, particle, precision=precision,
                  accel=rng.choice(["gmres", "bicgstab"]), tol=1e-6, bcz=rng.choice([0, 1]))
    elif kind == "dg2":
        c = _grid("", (log(12, 40), log(12, 40)), rng.randint(1, 2), rng.choice([4, 6]), rng.randint(1, 3), "photon",
                  order=2, entry=rng.choice(["dropin", "resident"]))
    else:
        c = {"kind": "serving", "count": rng.randint(3, 12), "max_cells": log(100, 600), "max_groups": rng.randint(12, 30),
             "max_side": rng.randint(34, 64), "precision": precision, "mix": rng.randint(0, 10 ** 6)}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
E_TOP = 2.0  # MeV


def _e_cut(groups):
    """The lower end of `groups` log-spaced groups as wide as those of the 40- and 80-group
    configurations (10 keV - 6 MeV, 1 keV - 20 MeV: 0.12 to 0.16 in the logarithm)."""
    return E_TOP * math.exp(-0.14 * groups)


def _settings(case, ndims):
    axes = ["x", "y", "z"][:ndims]
    csd = case["particle"] != "photon"
    kind, order = ("DD", 1) if case["order"] == 1 else ("DG", case["order"])
    names = axes + (["E"] if csd else [])
    return SN.SNSettings(
        solver_type="BFP" if csd else "BTE", quadrature_type="gauss-legendre" if ndims == 1 else "carlson",
        quadrature_order=case["sn"], legendre_order=case["legendre"], scheme_type={a: kind for a in names},
        scheme_order={a: order for a in names}, acceleration=case["accel"], convergence_criterion=case["tol"],
        angular_fokker_planck="galerkin")


def _slab_tables(case, seed):
    rng = np.random.default_rng(seed)
    nx, csd = case["cells"], case["particle"] != "photon"
    mats = np.ones(nx, dtype=np.int32)
    a = int(rng.integers(nx // 5, nx // 2))
    mats[a:a + nx // 5 + 1] = 2
    xs = W.synthetic_xs(case["groups"], 2, case["legendre"], seed, csd=csd, e_top=E_TOP,
                         e_cut=_e_cut(case["groups"]))
    return W.slab_tables(nx, np.full(nx, 10.0 / nx), mats, case["groups"], 2, seed, _settings(case, 1), case["legendre"],
                         beam_group=0, csd=csd, precision=case["precision"], xs=xs)


def _grid_tables(case, seed):
    """(tables, source set or None): 2D grids carry a beam on the left face (photons) or a source
    box as dense arrays; 3D grids give their source box as a definition, built on the device."""
    rng = np.random.default_rng(seed)
    ndims = 3 if case["nz"] else 2
    ns = [case["nx"], case["ny"], case["nz"]][:ndims]
    csd = case["particle"] != "photon"
    length = 16.0
    widths = [np.full(n, length / n) for n in ns]
    mats = np.ones(ns, dtype=np.int32)
    for tag in (2, 3):
        lo = [int(rng.integers(0, n - max(1, n // 4) + 1)) for n in ns]
        mats[tuple(slice(o, o + max(1, n // 4)) for o, n in zip(lo, ns))] = tag
    sn = _settings(case, ndims)
    xs = W.synthetic_xs(case["groups"], 3, case["legendre"], seed, csd=csd, e_top=E_TOP,
                         e_cut=_e_cut(case["groups"]))
    box = {a: (length / 2 - 2.0, length / 2 + 2.0) for a in range(ndims)}
    bc = (0, 0, 0, 0, case["bcz"], 0)
    if ndims == 2:
        beam = None if csd else ("X-", 0, (1.0, 0.0, 0.0), {1: (6.0, 10.0)})
        return W.grid_tables(2, ns, widths, mats, case["groups"], 3, seed, sn, case["legendre"], beam=beam,
                             volume=(0, box) if csd else None, bc=bc, csd=csd, precision=case["precision"], xs=xs), None
    tabs = SN.prepare_sn_tables(xs, 3, ns, widths, mats.reshape(ns, order="F"), list(bc), sn, precision=case["precision"])
    defs = W.grid_source_definitions(3, None, (0, box))
    sset = SRC.SourceSet(sn, 3, [SRC.positions_of(w) for w in widths], defs["volume"], defs["surface"],
                         np_surf=tabs["np_surf"])
    tabs["np_source"] = sset.np_source
    tabs["box"] = box
    return tabs, sset


def _stream(case, seed):
    """The requests of a batch or burst, each the list of its particle solves, as the serving
    configuration mixes them: slabs of S8-S32, P1-P7 and 1-5 layers (7 in 10 of a burst, all of a
    batch) or square grids of S4-S8, a photon alone or photon, electron and positron. The layouts
    belong to the case; the cross sections and the materials of the layers come from the seed."""
    lay, val = np.random.default_rng(case["mix"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        grid = case["kind"] == "serving" and lay.uniform() >= 0.7
        parts = ["photon"] if lay.uniform() < 0.5 else ["photon", "electron", "positron"]
        if case["kind"] == "batch":
            parts = parts[-1:]
        c = {"groups": int(lay.integers(case["max_groups"] // 2, case["max_groups"] + 1)), "order": 1, "accel": "gmres",
             "tol": 1e-7, "precision": case["precision"], "legendre": int(lay.integers(1, 4 if grid else 8))}
        if grid:
            n, c["sn"] = int(lay.integers(24, case["max_side"] + 1)), int(lay.choice([4, 6, 8]))
        else:
            n, c["sn"] = int(lay.integers(50, case["max_cells"] + 1)), int(lay.choice([8, 16, 32]))
        cuts = sorted(lay.choice(np.arange(1, n), size=int(lay.integers(0, 5)), replace=False).tolist()) + [n]
        width = lay.uniform(4.0, 16.0)
        mats = np.ones((n, n) if grid else n, dtype=np.int32)
        start = 0
        for k in cuts:
            mats[start:k] = int(val.integers(1, 5))
            start = k
        solves = []
        for part in parts:
            c["particle"], csd = part, part != "photon"
            if grid and csd:
                c["precision"] = "fp64"  # the serving stream keeps its grids in FP64
            sn, xs_seed = _settings(c, 2 if grid else 1), int(val.integers(0, 2 ** 31 - 1))
            xs = W.synthetic_xs(c["groups"], 4, c["legendre"], xs_seed, csd=csd, e_top=E_TOP, e_cut=_e_cut(c["groups"]))
            if grid:
                solves.append(W.grid_tables(2, [n, n], [np.full(n, width / n)] * 2, mats, c["groups"], 4, 0, sn,
                                            c["legendre"], beam=("X-", 0, (1.0, 0.0, 0.0), {1: (width / 4, 3 * width / 4)}),
                                            csd=csd, precision=c["precision"], xs=xs))
            else:
                solves.append(W.slab_tables(n, np.full(n, width / n), mats, c["groups"], 4, 0, sn, c["legendre"],
                                            beam_group=0, csd=csd, precision=c["precision"], xs=xs))
        out.append(solves)
    return out


def _coupled(case, seed):
    return W.coupled_particles(1, seed=seed % 100003, ng=case["groups"], n=case["cells"], photon_quad=case["sn"],
                               L=case["legendre"])


class _Resident:
    """Uploaded problems with their host result buffers; released with the object."""

    def __init__(self, items):
        self.ctx = SN.default_context()
        self.packs, self.results, self.handles = [], [], []
        for tabs, sset in items:
            pp = PackedProblem(tabs, pinned=True)
            self.handles.append(self.ctx.upload(pp) if sset is None else self.ctx.upload_sources(pp, sset)[0])
            self.packs.append(pp)
            self.results.append(ResultBuffers(pp, pinned=True))
        weakref.finalize(self, _release, self.ctx, list(self.handles))


def _release(ctx, handles):
    for h in handles:
        ctx.release(h)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"kind": kind, "plan": _Resident([(t, None) for q in _stream(case, seed) for t in q])}
    if kind == "serving":
        return {"kind": kind, "ctx": SN.default_context(),
                "tables": _stream(case, seed)}
    if kind == "coupled":
        parts, couplings = _coupled(case, seed)
        return {"kind": kind, "parts": parts, "couplings": couplings}
    tabs, sset = (_slab_tables(case, seed), None) if kind == "slab" else _grid_tables(case, seed)
    if case["entry"] == "dropin":
        return {"kind": "dropin", "tables": tabs}
    return {"kind": "resident", "plan": _Resident([(tabs, sset)])}


def _record(r):
    """What a solve gives back: the flux moments, the cutoff flux (CSD solvers), and the
    iterations and passes it took."""
    return {"flux": r.flux, "cutoff": r.flux_cutoff, "iters": r.group_iters, "passes": r.passes}


def run(state):
    kind = state["kind"]
    if kind == "dropin":
        return _record(SN.compute_flux_tables(state["tables"]))
    if kind == "resident":
        p = state["plan"]
        p.ctx.solve(p.handles[0])
        p.ctx.download(p.handles[0], p.results[0])
        return _record(p.results[0])
    if kind == "batch":
        p = state["plan"]
        p.ctx.solve_batch(p.handles)
        for h, r in zip(p.handles, p.results):
            p.ctx.download(h, r)
        return _joined([_record(r) for r in p.results])
    if kind == "serving":
        reqs = [SV.Request(i, t, 0.0) for i, t in enumerate(state["tables"])]
        SV.ServingLoop(state["ctx"]).run(reqs)
        return _joined([_record(r) for q in reqs for r in q.results])
    out = TR.transport_tables(state["parts"], state["couplings"], ngen_max=12, eps_gen=1e-6)
    res = _joined([_record(r) for r in out.fluxes])
    res["generations"] = out.generations
    return res


def _joined(records):
    """Several solves' records as one: every value of every solve, end to end."""
    def flat(key):
        return np.concatenate([np.ravel(r[key], order="K") for r in records if r[key] is not None] or [np.zeros(0)])

    return {"flux": flat("flux"), "cutoff": flat("cutoff"), "iters": flat("iters"),
            "passes": np.array([r["passes"] for r in records])}


# ------------------------------------------------------------------------------------------
# what a pass through a case cannot do without
# ------------------------------------------------------------------------------------------
PASSES = 8  # transport passes per group that the in-group iteration takes at the least here


def _shape(case):
    """(groups, moments, directions, cells, cell moments, CSD) of one solve of the case."""
    csd = case.get("particle", "photon") != "photon"
    if case["kind"] == "slab":
        nd, cells, axes = case["sn"], case["cells"], 1
        np_ = nd
    else:
        n, cells = case["sn"], case["nx"] * case["ny"] * max(1, case["nz"])
        nd = n * (n + 2)  # level-symmetric directions of the sphere
        np_, axes = nd, 3 if case["nz"] else 2
    return case["groups"], np_, nd, cells, case["order"] ** (axes + csd), csd


def _solve_work(ng, np_, nd, cells, nm, csd):
    col = float(cells) * nm
    out = 8.0 * ng * np_ * col + (8.0 * np_ * col if csd else 0.0)
    per_pass = 2.0 * 2.0 * nd * np_ * col + 12.0 * nd * col * nm
    return out, PASSES * ng * per_pass


def work(case):
    kind = case["kind"]
    if kind in ("slab", "grid"):
        b, f = _solve_work(*_shape(case))
    elif kind == "coupled":
        b, f = _solve_work(case["groups"], case["sn"], case["sn"], case["cells"], 4, True)
        b, f = 3 * b, 3 * 4 * f  # three particles, some generations
    else:  # mean sizes of the seeded streams
        ng, cells = (10 + case["max_groups"]) / 2, (50 + case["max_cells"]) / 2
        b, f = _solve_work(ng, 6, 30, cells, 1, True)
        n = case["count"] * (2 if kind == "serving" else 1)
        b, f = n * b, n * f
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------------
# the same equations in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------
class _Budget:
    """Sweep steps (a step is a handful of torch calls) that an exact value may spend."""

    def __init__(self, steps=90_000):
        self.left = steps

    def take(self, steps):
        self.left -= steps
        return self.left >= 0


def _moment_lists(ndims, csd, order, fc):
    """Cell moments as tuples (x, y, z, E), E fastest, and per axis the face moment of each."""
    axes = ([3] if csd else []) + list(range(ndims))
    o = [order[a] for a in axes]
    tup = []
    for c in range(int(np.prod(o))):
        t, r = [], c
        for n in o:
            t.append(r % n + 1)
            r //= n
        tup.append(t)
    if not fc:
        tup = [t for t in tup if sum(v > 1 for v in t) < 2]
        tup.sort(key=lambda t: _flat(o, t, False))
    face, nface = {}, {}
    for i, a in enumerate(axes):
        so = o[:i] + o[i + 1:]
        face[a] = [_flat(so, t[:i] + t[i + 1:], fc) for t in tup]
        nface[a] = int(np.prod(so)) if fc else 1 + sum(n - 1 for n in so)
    full = []
    for t in tup:
        f = [1, 1, 1, 1]
        for i, a in enumerate(axes):
            f[a] = t[i]
        full.append(f)
    return full, face, nface


def _flat(orders, t, fc):
    if fc:
        i, stride = 0, 1
        for n, v in zip(orders, t):
            i += (v - 1) * stride
            stride *= n
        return i
    off = 1
    for n, v in zip(orders, t):
        if v > 1:
            return off + v - 2
        off += n - 1
    return 0


class _Exact:
    """One SN solve: the group loop with every in-group problem solved to rounding."""

    def __init__(self, t, volume=None, budget=None, extra=None):
        self.t, self.budget, self.extra = t, budget or _Budget(), extra
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.nd, self.P, self.nps, self.ng = t["nd"], t["np"], t["np_surf"], t["ng"]
        self.ndims = t["ndims"]
        self.ns = [int(v) for v in t["ns"]] + [1] * (3 - len(t["ns"]))
        self.csd = t["solver_type"] >= 2
        self.fp = t["solver_type"] == 2
        self.tup, self.face, self.nface = _moment_lists(self.ndims, self.csd, t["order"], t["is_fc"])
        self.nm = len(self.tup)
        self.ne = self.nface[3] if self.csd else 1
        self.mn, self.dn = self._t(t["mn"]), self._t(t["dn"])
        self.mnfp = self._t(np.asarray(t["mn"]) @ np.asarray(t["fp"])) if self.fp else None
        self.mat = torch.as_tensor(np.asarray(t["mat"]).reshape(self.ns, order="F").astype(np.int64) - 1, device=self.dev)
        self.om = [np.asarray(o, dtype=float) for o in t["omega"]]
        self.vol = volume if volume is not None else t.get("volume_sources")
        self._closures()
        self._surface_rows()
        self._flips()

    def _t(self, a):
        return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=self.dev)

    def _closures(self):
        t, nm, C = self.t, self.nm, self.t["cc"]
        m1 = lambda k: 1.0 if k % 2 == 0 else -1.0  # noqa: E731
        self.G, self.Gs, self.Go = [], [], []
        for a in range(self.ndims):
            w, nf = t["w_axis"][a], self.nface[a]
            G, Gs, Go = np.zeros((self.nd, nm, nm)), np.zeros((self.nd, nm, nf)), np.zeros((self.nd, nf, nm))
            for n in range(self.nd):
                s = float(np.sign(self.om[a][n]))
                for i in range(nm):
                    for j in range(nm):
                        if any(k != a and self.tup[i][k] != self.tup[j][k] for k in range(4)):
                            continue
                        ia, ja = self.tup[i][a], self.tup[j][a]
                        v = C[ia - 1] * s ** (ia - 1) * C[ja - 1] * s ** (ja - 1) * w[ja]
                        if ia > ja:
                            v -= C[ia - 1] * s * C[ja - 1] * (1.0 - m1(ia - ja))
                        G[n, i, j] = v
                for j in range(nm):
                    ja, f = self.tup[j][a], self.face[a][j]
                    Gs[n, j, f] = -C[ja - 1] * (s ** (ja - 1) * w[0] - (-s) ** (ja - 1))
                    Go[n, f, j] = C[ja - 1] * s ** (ja - 1) * w[ja]
            self.G.append(self._t(G)); self.Gs.append(self._t(Gs)); self.Go.append(self._t(Go))
        if self.csd:
            oE, wE, ww = t["order"][3], t["w_axis"][3], np.asarray(t["ww"])
            K, B = np.zeros((oE, nm, nm)), np.zeros((nm, nm))
            A1, A2, E = np.zeros((nm, self.ne)), np.zeros((nm, self.ne)), np.zeros((self.ne, nm))
            for i in range(nm):
                for j in range(nm):
                    if any(self.tup[i][d] != self.tup[j][d] for d in range(self.ndims)):
                        continue
                    iE, jE = self.tup[i][3], self.tup[j][3]
                    for kE in range(1, iE):
                        for wi in range(1, oE + 1):
                            K[wi - 1, i, j] += (C[iE - 1] * C[jE - 1] * C[kE - 1] * C[wi - 1] * (1.0 - m1(iE - kE))
                                                * ww[jE - 1, kE - 1, wi - 1])
                    B[i, j] = C[iE - 1] * m1(iE - 1) * C[jE - 1] * m1(jE - 1) * wE[jE]
            for j in range(nm):
                jE, e = self.tup[j][3], self.face[3][j]
                A1[j, e] = C[jE - 1] * m1(jE - 1) * wE[0]
                A2[j, e] = C[jE - 1]
                E[e, j] = C[jE - 1] * m1(jE - 1) * wE[jE]
            self.K, self.B, self.EA, self.EB, self.EO = (self._t(x) for x in (K, B, A1, A2, E))

    def _surface_rows(self):
        t = self.t
        self.rm, self.rd, self.fwd = [], [], []
        for a in range(self.ndims):
            rm, rd = np.zeros((self.nd, self.nps)), np.zeros((self.nd, self.nps))
            for n in range(self.nd):
                for f in (2 * a, 2 * a + 1):
                    k = int(t["n_to_nplus"][f][n])
                    if k:
                        rm[n], rd[n] = t["mn_surf"][f][k - 1, :], t["dn_surf"][f][:, k - 1]
                        break
            self.rm.append(self._t(rm)); self.rd.append(self._t(rd))
            self.fwd.append(torch.as_tensor(self.om[a] >= 0.0, device=self.dev))

    def _flips(self):
        groups = {}
        for n in range(self.nd):
            key = tuple(a for a in range(self.ndims) if self.om[a][n] < 0.0)
            groups.setdefault(key, []).append(n)
        self.groups = [(list(k), torch.as_tensor(v, device=self.dev)) for k, v in groups.items()]
        X, Y, Z = self.ns
        i, j, k = torch.meshgrid(torch.arange(X), torch.arange(Y), torch.arange(Z), indexing="ij")
        s = (i + j + k).reshape(-1)
        order = torch.argsort(s, stable=True)
        cuts = torch.searchsorted(s[order].contiguous(), torch.arange(X + Y + Z - 1))
        cuts = cuts.tolist() + [X * Y * Z]
        flat = lambda v: v.reshape(-1)[order].to(self.dev)  # noqa: E731
        I, J, Kk = flat(i), flat(j), flat(k)
        self.planes = [(I[a:b], J[a:b], Kk[a:b]) for a, b in zip(cuts[:-1], cuts[1:])]
        self.matf = self._flip(self.mat[..., None].expand(X, Y, Z, self.nd))
        self.inv = []  # per axis: 1 / width by flipped index and direction
        for a in range(self.ndims):
            w = self._t(1.0 / np.asarray(self.t["ds"][a], dtype=float))
            v = w[:, None].expand(self.ns[a], self.nd).clone()
            neg = ~self.fwd[a]
            v[:, neg] = torch.flip(w, [0])[:, None].expand(self.ns[a], int(neg.sum()))
            self.inv.append(v * self._t(np.abs(self.om[a]))[None, :])

    def _flip(self, v, axes=(0, 1, 2), at=3):
        """Turns v[x, y, z, n, ...] into (or out of) each direction's sweep order; `axes` are the
        geometry axes of the leading dimensions."""
        out = v.clone()
        for key, n in self.groups:
            dims = [axes.index(a) for a in key if a in axes]
            if dims:
                out.index_copy_(at, n, torch.flip(v.index_select(at, n), dims))
        return out

    def sweep(self, q, fin, fe):
        """q [X,Y,Z,nd,nm,B], fin per axis [.., .., nd, nf, B] (sweep order), fe [X,Y,Z,nd,ne,B] or
        None: the angular flux, outgoing faces per axis and energy-face flux."""
        F = [f.clone() for f in fin]
        psi = torch.empty_like(q)
        feo = torch.empty_like(fe) if fe is not None else None
        for I, J, K in self.planes:
            at = [(J, K), (I, K), (I, J)]
            m = self.matf[I, J, K]
            S, rhs = self.S0[m], q[I, J, K]
            ins = []
            for a in range(self.ndims):
                h = self.inv[a][(I, J, K)[a]]
                f = F[a][at[a]]
                ins.append(f)
                S = S + h[..., None, None] * self.G[a]
                rhs = rhs + h[..., None, None] * (self.Gs[a] @ f)
            if fe is not None:
                fi = fe[I, J, K]
                rhs = rhs - self.ES[m] @ fi
            v = rhs / S if self.nm == 1 else torch.linalg.solve(S, rhs)
            psi[I, J, K] = v
            for a in range(self.ndims):
                F[a][at[a]] = self.t["w_axis"][a][0] * ins[a] + self.Go[a] @ v
            if fe is not None:
                feo[I, J, K] = self.t["w_axis"][3][0] * fi + self.EO @ v
        return psi, F, feo

    def group(self, ig):
        """Sets the constants of group ig."""
        t, nm = self.t, self.nm
        eye = torch.eye(nm, dtype=torch.float64, device=self.dev)
        S0 = self._t(t["sigma_t"][ig])[:, None, None] * eye
        if self.csd:
            de = float(t["e_width"][ig])
            sp, sm = self._t(t["s_plus"][ig]) / de, self._t(t["s_minus"][ig]) / de
            S0 = S0 + sp[:, None, None] * self.B
            for w in range(self.K.shape[0]):
                S0 = S0 + (self._t(t["s_mom"][ig][:, w]) / de)[:, None, None] * self.K[w]
            self.ES = sp[:, None, None] * self.EA - sm[:, None, None] * self.EB
        self.S0 = S0
        pl = np.asarray(t["pl"])
        self.ks = self._t(np.asarray(t["sigma_s"])[:, ig, ig, :][:, pl])[self.mat]        # [X,Y,Z,P]
        self.kt = self._t(t["t_mom"][ig])[self.mat] if self.fp else None                  # [X,Y,Z]
        if self.ndims == 1:
            self._operator()

    def _operator(self):
        """1D: the sweep's response to every unit source and incoming face, once per group."""
        X, nd, nm, nf = self.ns[0], self.nd, self.nm, self.nface[0]
        B = X * nm + nf
        q = torch.zeros((X, 1, 1, nd, nm, B), dtype=torch.float64, device=self.dev)
        e = torch.eye(X * nm, dtype=torch.float64, device=self.dev).reshape(X, nm, X * nm)
        q[:, 0, 0, :, :, :X * nm] = e[:, None].expand(X, nd, nm, X * nm)
        f = torch.zeros((1, 1, nd, nf, B), dtype=torch.float64, device=self.dev)
        f[..., X * nm:] = torch.eye(nf, dtype=torch.float64, device=self.dev)
        psi, F, _ = self.sweep(q, [f], None)
        self.Tp = psi[:, 0, 0].permute(1, 0, 2, 3).reshape(nd, X * nm, B)
        self.Tf = F[0][0, 0]

    def _boundary_in(self, a, b, ig, source):
        """Incoming faces of axis a in face order [.., .., nd, nf] from the out-moments
        b [fa, fb, side, nf, nps] of the last pass and the surface sources."""
        t = self.t
        dims = [d for d in range(3) if d != a]
        out = torch.zeros((self.ns[dims[0]], self.ns[dims[1]], self.nd, self.nface[a]), dtype=torch.float64, device=self.dev)
        for side in (0, 1):
            n = self.fwd[a] if side == 0 else ~self.fwd[a]
            bcv = int(t["bc"][2 * a + side])
            if bcv:
                src = b[:, :, side if bcv == 1 else 1 - side]
                out[:, :, n] += torch.einsum("np,uvfp->uvnf", self.rm[a][n], src)
            s = t["surface_sources"][2 * a + side] if source else None
            if s is not None:
                v = self._t(np.asarray(s)[ig].reshape(s.shape[1], self.ns[dims[0]], self.ns[dims[1]], order="F"))
                out[:, :, n, 0] += torch.einsum("np,puv->uvn", self.rm[a][n][:, :s.shape[1]], v)
        return out

    def _pass(self, phi, b, ig, qn, fe):
        """T(z): qn None is the homogeneous operator. phi [X,Y,Z,nm,P]."""
        src = torch.einsum("xyzmp,np->xyznm", phi * self.ks[..., None, :], self.mn)
        if self.fp:
            src = src + torch.einsum("xyzmp,np->xyznm", phi * self.kt[..., None, None], self.mnfp)
        if qn is not None:
            src = src + qn
        src = self._flip(src)
        fin = []
        for a in range(self.ndims):
            dims = [d for d in range(3) if d != a]
            fin.append(self._flip(self._boundary_in(a, b[a], ig, qn is not None), axes=tuple(dims), at=2))
        if self.ndims == 1:
            X, nm = self.ns[0], self.nm
            v = torch.cat([src[:, 0, 0].permute(1, 0, 2).reshape(self.nd, X * nm), fin[0][0, 0]], dim=1)[..., None]
            psi = (self.Tp @ v).reshape(self.nd, X, nm).permute(1, 0, 2)[:, None, None]
            F = [(self.Tf @ v)[None, None]]
            feo = None
            if fe is not None:
                zero = torch.zeros_like(src)[..., None]
                p2, F2, feo = self.sweep(zero, [torch.zeros_like(fin[0])[..., None]], fe[..., None])
                feo = feo[..., 0]
                # the sweep is linear: its answer to the incoming energy flux, then the rest of it
                psi = psi + p2[..., 0]
                F = [F[0] + F2[0]]
                feo = feo + torch.einsum("em,xyznm->xyzne", self.EO, psi - p2[..., 0])
            psi = psi[..., None]
        else:
            psi, F, feo = self.sweep(src[..., None], [f[..., None] for f in fin], None if fe is None else fe[..., None])
            if feo is not None:
                feo = feo[..., 0]
        psi = self._flip(psi[..., 0])
        out = torch.einsum("pn,xyznm->xyzmp", self.dn, psi)
        bo = []
        for a in range(self.ndims):
            dims = [d for d in range(3) if d != a]
            ex = self._flip(F[a][..., 0], axes=tuple(dims), at=2)
            sides = []
            for side in (0, 1):
                n = ~self.fwd[a] if side == 0 else self.fwd[a]
                sides.append(torch.einsum("uvnf,np->uvfp", ex[:, :, n], self.rd[a][n]))
            bo.append(torch.stack(sides, dim=2))
        return out, bo, feo

    def solve(self):
        X, Y, Z = self.ns
        nm, P, dev = self.nm, self.P, self.dev
        steps = self.ng * (X if self.ndims == 1 else 30 * (X + Y + Z))
        if not self.budget.take(steps * (2 if self.csd and self.ndims == 1 else 1)):
            return None
        pl = np.asarray(self.t["pl"])
        flux = torch.zeros((self.ng, X, Y, Z, nm, P), dtype=torch.float64, device=dev)
        fe = torch.zeros((X, Y, Z, self.nd, self.ne), dtype=torch.float64, device=dev) if self.csd else None
        bz = [torch.zeros((self.ns[[1, 0, 0][a]], self.ns[[2, 2, 1][a]], 2, self.nface[a], self.nps), dtype=torch.float64,
                          device=dev) for a in range(self.ndims)]
        zero = torch.zeros((X, Y, Z, nm, P), dtype=torch.float64, device=dev)

        def pack(phi, b):
            return torch.cat([phi.reshape(-1)] + [x.reshape(-1) for x in b])

        def unpack(v):
            phi, b, o = v[:zero.numel()].reshape(zero.shape), [], zero.numel()
            for x in bz:
                b.append(v[o:o + x.numel()].reshape(x.shape))
                o += x.numel()
            return phi, b

        for ig in range(self.ng):
            self.group(ig)
            q = torch.zeros_like(zero)
            for gi in range(ig):
                ss = self._t(np.asarray(self.t["sigma_s"])[:, gi, ig, :][:, pl])[self.mat]
                q += ss[..., None, :] * flux[gi]
            if self.vol is not None:
                q += self._t(np.asarray(self.vol[ig]).transpose(2, 3, 4, 1, 0))
            if self.extra is not None:
                q += self.extra[ig]
            qn = torch.einsum("xyzmp,np->xyznm", q, self.mn)
            if self.csd and ig > 0:
                fe = fe * float(self.t["e_width"][ig]) / float(self.t["e_width"][ig - 1])
            fef = self._flip(fe) if self.csd else None
            o, b, feo = self._pass(zero, bz, ig, qn, fef)
            c = pack(o, b)

            def mul(v):
                o, b, _ = self._pass(*unpack(v), ig, None, None)
                return v - pack(o, b)

            z = _gmres(mul, c)
            o, b, feo = self._pass(*unpack(z), ig, qn, fef)
            flux[ig] = o
            if self.csd:
                fe = self._flip(feo)
        cut = None
        if self.csd:
            cut = torch.zeros((P, nm, X, Y, Z), dtype=torch.float64, device=dev)
            cut[:, :self.ne] = torch.einsum("pn,xyzne->pexyz", self.dn, fe)
        self.raw = flux
        return {"flux": flux.permute(0, 5, 4, 1, 2, 3), "cutoff": cut, "iters": None, "passes": None}


def _gmres(mul, c, tol=1e-13, most=80):
    """(I − A) z = c to rounding: full orthogonalisation twice, restarted once at `most`."""
    bn = float(c.norm())
    z = torch.zeros_like(c)
    if bn == 0.0:
        return z
    for _ in range(2):
        r = c - mul(z) if float(z.norm()) > 0 else c.clone()
        beta = float(r.norm())
        if beta <= tol * bn:
            return z
        V, H = [r / beta], np.zeros((most + 1, most))
        for j in range(most):
            w = mul(V[j])
            B = torch.stack(V)
            for _ in range(2):
                h = B @ w
                w = w - B.T @ h
                H[:j + 1, j] += h.cpu().numpy()
            H[j + 1, j] = float(w.norm())
            e = np.zeros(j + 2)
            e[0] = beta
            y, *_ = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)
            res = np.linalg.norm(H[:j + 2, :j + 1] @ y - e)
            if res <= tol * bn or H[j + 1, j] == 0.0:
                break
            V.append(w / H[j + 1, j])
        z = z + torch.stack(V[:len(y)]).T @ torch.as_tensor(y, device=c.device)
    return z


def _box_source(tabs):
    """The dense volume sources of a 3D case's source box: one per voxel whose centre is inside."""
    v = np.zeros((tabs["ng"], tabs["np"], 1, *tabs["ns"]))
    inside = np.ones(tabs["ns"], dtype=bool)
    for a, w in enumerate(tabs["ds"]):
        x = np.cumsum(w) - np.asarray(w) / 2
        lo, hi = tabs["box"][a]
        shape = [1, 1, 1]
        shape[a] = -1
        inside &= ((x >= lo) & (x <= hi)).reshape(shape)
    v[0, 0, 0][inside] = 1.0
    return v


def _exact_joined(outs):
    """Joined as run joins them; solves that were left out make the whole without a value."""
    if any(o is None for o in outs):
        return None

    def flat(key):
        parts = [o[key] for o in outs if o[key] is not None]
        # the buffers of a solve are column-major
        return torch.cat([p.permute(*reversed(range(p.ndim))).reshape(-1) for p in parts]) if parts else np.zeros(0)

    return {"flux": flat("flux"), "cutoff": flat("cutoff"), "iters": None, "passes": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "slab":
        return _Exact(_slab_tables(case, seed)).solve()
    if kind == "grid":
        tabs, sset = _grid_tables(case, seed)
        return _Exact(tabs, _box_source(tabs) if sset is not None else None).solve()
    budget = _Budget()
    if kind == "coupled":
        return _exact_coupled(case, seed)
    tabs = [t for q in _stream(case, seed) for t in q]
    outs = []
    for t in tabs:
        outs.append(_Exact(t, budget=budget).solve() if budget.left > 0 else None)
        if outs[-1] is None:
            return None
    return _exact_joined(outs)


def _exact_coupled(case, seed):
    parts, couplings = _coupled(case, seed)
    n = len(parts)
    solvers = [_Exact(t) for t in parts]
    total, cut, pend, last = [None] * n, [None] * n, [None] * n, [None] * n
    generations = 0
    for gen in range(12):
        generations += 1
        before = [None if f is None else f.clone() for f in total]
        for i in range(n):
            s = solvers[i]
            if gen > 0:
                s.vol = None
                s.t = dict(s.t, surface_sources=[None] * 6)
            s.extra, pend[i] = pend[i], None
            r = s.solve()
            if r is None:
                return None
            flux = s.raw
            total[i] = flux.clone() if total[i] is None else total[i] + flux
            if r["cutoff"] is not None:
                cut[i] = r["cutoff"].clone() if cut[i] is None else cut[i] + r["cutoff"]
            for j in range(n):
                if j == i or (i, j) not in couplings:
                    continue
                c = couplings[(i, j)]
                pl = np.asarray(parts[i]["pl"])
                ss = s._t(np.asarray(c.sigma_s)[:, :, :, pl])[s.mat]              # [X,Y,Z,gi,gf,P]
                q = torch.einsum("xyzghp,gxyzmp->hxyzmp", ss, flux)
                src = torch.zeros((parts[j]["ng"], *s.ns, len(c.moment_map), parts[j]["np"]), dtype=torch.float64,
                                  device=s.dev)
                tr = s._t(c.transfer)
                for k, mk in enumerate(c.moment_map):
                    if mk:
                        src[..., k, :] = q[..., int(mk) - 1, :] @ tr.T
                pend[j] = src if pend[j] is None else pend[j] + src
        if gen > 0:
            eps = 0.0
            for i in range(n):
                a, b = total[i][..., 0, 0], before[i][..., 0, 0]
                eps = max(eps, float(((a - b).abs() / a.abs().clamp_min(np.finfo(float).eps)).max()))
            if eps < 1e-6:
                break
    out = _exact_joined([{"flux": f.permute(0, 5, 4, 1, 2, 3), "cutoff": c} for f, c in zip(total, cut)])
    out["generations"] = None
    return out
