"""The engine's work as its users run it, as cases that can be timed and checked.

Each case goes through the public host API: `thrid_b200.pgk.PgkEngine` for one
system, `thrid_b200.serve.ReplicaServer` for a batch of them.  The listed sizes
are the configurations of `thrid_b200/systems.py` and of `bench.py`; `draw`
gives more of the same ranges, ragged molecule counts and grids among them.

A case's `call`:
  force   one single-point evaluation from host coordinates: pair list, forces,
          energies and virials (a driver that keeps the integrator on the host,
          an energy check of a stored frame)
  md      steps 0..n of NVE, NHC or MTK dynamics from an uploaded state to a
          downloaded one, one pair-list period long (the production run)
  host    the same, but the host owns the state and drives single steps
  hf      dynamics with the heat flux of every step streamed out, with or
          without region Langevin thermostats (Green-Kubo and NEMD runs)
  ewk     the per-atom standard-Ewald term of the bulk heat flux
  serve   a batch of independent replicas through the replica server

Results of the mixed-precision engine leave in single precision, as a
trajectory or force file holds them; the FP64 engine's stay in double.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from thrid_b200 import abi
from thrid_b200 import systems as S
from thrid_b200.pgk import PgkEngine
from thrid_b200.serve import ReplicaServer

DT = S.fs_to_reduced(1.0)
GRIDS = (16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 120, 125,
         128)


def _box(kind, nside, nmol=0, spacing=0.0, prec="mixed", grid=0, order=4, rcut=0.0):
    """The fields that describe one box of nmol (0: nside^3) molecules."""
    return {"kind": kind, "nside": nside, "nmol": nmol or nside ** 3,
            "spacing": spacing or {"water": 3.10375, "propanol": 5.2, "butane": 5.2}[kind],
            "prec": prec, "grid": grid, "order": order, "rcut": rcut}


def listed():
    return [
        # the smallest call: one energy of 512 rigid waters in double precision
        {"name": "force_water1536_fp64", "call": "force", **_box("water", 8, prec="fp64", grid=32, rcut=10.0)},
        # single-point of the 12,000-atom propanol box, as a host-side driver asks for it
        {"name": "force_propanol12000", "call": "force", **_box("propanol", 10, grid=64, rcut=12.0)},
        # small production run, launch-bound: 512 rigid waters, NVE
        {"name": "nve_water1536", "call": "md", "ens": "nve", "steps": 49, **_box("water", 8, grid=32, rcut=10.0)},
        # the same in the all-FP64 engine (the plain method)
        {"name": "nve_water1536_fp64", "call": "md", "ens": "nve", "steps": 49,
         **_box("water", 8, prec="fp64", grid=32, rcut=10.0)},
        # ordinary production run: 1000 flexible 1-propanol, Nose-Hoover chains
        {"name": "nhc_propanol12000", "call": "md", "ens": "nhc", "steps": 49, **_box("propanol", 10, grid=64, rcut=12.0)},
        # the host program owns the state and asks for one step at a time
        {"name": "host_propanol12000", "call": "host", "ens": "nhc", "steps": 12,
         **_box("propanol", 10, grid=64, rcut=12.0)},
        # the largest: 200,004 atoms of butane at constant pressure
        {"name": "mtk_butane200004", "call": "md", "ens": "mtk", "steps": 49,
         **_box("butane", 25, 14286, grid=128, order=5, rcut=12.0)},
        {"name": "mtk_butane200004_fp64", "call": "md", "ens": "mtk", "steps": 9,
         **_box("butane", 25, 14286, prec="fp64", grid=128, order=5, rcut=12.0)},
        # heat flow through a water slab with propanol faces, hot and cold Langevin layers
        {"name": "hf_slab43200", "call": "hf", "kind": "slab", "layers": 32, "prec": "mixed", "steps": 10},
        # Green-Kubo replica: J_z(t) of a water box every step (short: the random lattice heats
        # up, and an atom that outruns the list's skin within a period changes the bare Coulomb flux)
        {"name": "hf_water8232", "call": "hf", "steps": 14, "regions": 1, **_box("water", 14, spacing=3.1, grid=48, rcut=10.0)},
        # per-atom standard-Ewald k-space term of 4096 waters
        {"name": "ewk_water12288", "call": "ewk", "kmax": 19, **_box("water", 16, prec="fp64", grid=32, rcut=10.0)},
        # a batch of uneven flexible replicas, continuous batching on eight slots
        {"name": "serve_8", "call": "serve", "replicas": 8, "low": 1500, "high": 12000, "steps": 300, "prec": "mixed"},
    ]


def _draw_box(rng, low, high, prec, kinds=("water", "propanol", "butane")):
    kind = rng.choice(kinds)
    per = {"water": 3, "propanol": 12, "butane": 14}[kind]
    spacing = {"water": 3.1, "propanol": 5.6, "butane": 5.4}[kind]
    want = math.exp(rng.uniform(math.log(low), math.log(high))) / per
    nside = max(7 if kind == "water" else 5, math.ceil(want ** (1.0 / 3.0)))
    nmol = nside ** 3 if kind == "water" else max(nside ** 3 - rng.randrange(nside * nside), 1)
    side = nside * spacing
    k = next((i for i, g in enumerate(GRIDS) if g >= 0.95 * side), len(GRIDS) - 1)
    grid = GRIDS[min(k + rng.randrange(2), len(GRIDS) - 1)]
    rcut = min(rng.uniform(9.0, 12.0), side / 2.0 - 2.2)
    return _box(kind, nside, nmol, spacing, prec, grid, rng.choice((4, 4, 5, 6)), round(rcut, 2))


def draw(rng):
    call = rng.choice(("force", "md", "md", "md", "host", "hf", "hf", "ewk", "serve"))
    prec = "fp64" if rng.random() < 0.3 else "mixed"
    if call == "force":
        return {"call": call, **_draw_box(rng, 1000, 60000, prec)}
    if call == "md":
        c = _draw_box(rng, 1000, 150000 if prec == "mixed" else 40000, prec)
        return {"call": call, "ens": rng.choice(("nve", "nhc", "mtk")), "steps": rng.randint(20, 49), **c}
    if call == "host":
        return {"call": call, "ens": rng.choice(("nve", "nhc")), "steps": rng.randint(5, 15),
                **_draw_box(rng, 1000, 30000, prec)}
    if call == "hf":
        if rng.random() < 0.4:
            return {"call": call, "kind": "slab", "layers": rng.randint(8, 28), "prec": prec, "steps": rng.randint(4, 9)}
        return {"call": call, "steps": rng.randint(6, 14), "regions": rng.choice((1, 1, rng.randint(2, 9))),
                **_draw_box(rng, 1500, 20000, prec, ("water", "water", "propanol"))}
    if call == "ewk":
        return {"call": call, "kmax": rng.randint(6, 18), **_draw_box(rng, 1500, 12000, "fp64", ("water", "propanol"))}
    return {"call": call, "replicas": rng.randint(3, 8), "low": 1200, "high": rng.randint(3000, 9000),
            "steps": rng.randint(80, 250), "prec": "mixed"}


# ---- the systems ---------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _topology(kind, nside, nmol, spacing, layers):
    """Molecules, force field and lattice of a box (the part that no seed changes)."""
    if kind == "slab":
        nwater = 250 * layers
        return S.slab_box(nlay_w=layers, nwater=nwater, nlay_p=max(2, layers // 4), nfft=(64, 64, 192))
    side = nside * spacing
    if kind == "water":
        return S.water_box(nside=nside, box=side)
    if kind == "propanol":
        return S.propanol_box(nside=nside, box=side, nmol=nmol)
    return S.butane_box(nmol=nmol, nside=nside, box=side)


def _system(case, seed):
    """One system: every molecule of the lattice moved by up to 0.05 A, Maxwell velocities."""
    base = _topology(case["kind"], case.get("nside", 0), case.get("nmol", 0), case.get("spacing", 0.0),
                     case.get("layers", 0))
    rng = np.random.default_rng(1000003 * seed + 17)
    mol = np.repeat(np.arange(base.nmole), np.diff(base.molept_index))
    shift = rng.uniform(-0.05, 0.05, (base.nmole, 3))[mol]
    temp = 250.0 if case["kind"] == "butane" else 300.0
    vel = rng.normal(size=(base.natom, 3)) * np.sqrt(S.kelvin_to_reduced(temp) / base.atmmass)[:, None]
    vel -= (base.atmmass[:, None] * vel).sum(axis=0) / base.atmmass.sum()
    p = dict(base.params, precision=abi.PREC_FP64 if case["prec"] == "fp64" else abi.PREC_MIXED)
    if case["kind"] != "slab":
        g, rc = case["grid"], case["rcut"]
        p.update(nfft1=g, nfft2=g, nfft3=g, pme_order=case["order"], rcut=rc, rrcut=rc, rcut_book=rc + 2.0,
                 alpha=3.3 / rc)
    return dataclasses.replace(base, atmcor=base.atmcor + shift, atmvel=vel, params=p)


def _md(s, ens, kind):
    t = S.kelvin_to_reduced(250.0 if kind == "butane" else 300.0)
    if ens == "nve":
        return abi.md_struct(DT, ifrattle=1, outinterval=0)
    return abi.md_struct(DT, mchain=3, text=t, tfreq=1.0e13 * S.TIMEREF, vfreq=0.2e12 * S.TIMEREF,
                         pext=S.pa_to_reduced(1.01325e5), pcont_axis=abi.PCONT_ANISO, degfree=s.degfree_all, ifrattle=1,
                         eps_rattle=1e-7, outinterval=0)


def _heat_flux(case, s):
    if case["kind"] == "slab":
        return s.regions["hf"]
    n, lz = case["regions"], float(s.box[2])
    return dict(regions=[(k * lz / n, (k + 1) * lz / n) for k in range(n)], heatfinterval=1)


def _replicas(case, seed):
    """Propanol and butane boxes of low..high atoms, spread evenly over the logarithm."""
    got = []
    for k in range(case["replicas"]):
        natom = case["low"] * (case["high"] / case["low"]) ** (k / max(1, case["replicas"] - 1))
        kind, per, spacing = (("propanol", 12, 5.6), ("butane", 14, 5.4))[k % 2]
        nside = max(5, round((natom / per) ** (1.0 / 3.0)))
        grid = next(g for g in GRIDS if g >= 0.95 * nside * spacing)
        rcut = min(10.0, nside * spacing / 2.0 - 2.2)
        got.append(_system(_box(kind, nside, 0, spacing, case["prec"], grid, 4, rcut), 100 * seed + k))
    return got


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


# ---- what is measured ----------------------------------------------------------------
def prepare(case, seed):
    if case["call"] == "serve":
        reps = _replicas(case, seed)
        return {"case": case, "server": ReplicaServer(max_slots=8), "systems": reps,
                "md": [_md(s, "nve", "") for s in reps]}
    s = _system(case, seed)
    eng = PgkEngine(s)
    st = {"case": case, "engine": eng, "system": s, "x": _pinned(s.atmcor), "v": _pinned(s.atmvel),
          "x_out": _pinned(s.atmcor), "v_out": _pinned(s.atmvel)}
    if case["call"] in ("md", "host", "hf"):
        st["md"] = _md(s, case.get("ens", "nve"), case["kind"])
    if case["call"] == "hf":
        eng.set_hf(_heat_flux(case, s))
    return st


def run(state):
    case = state["case"]
    out = np.float32 if case["prec"] == "mixed" else np.float64
    if case["call"] == "serve":
        srv = state["server"]
        ids = [srv.submit(s, md, nsteps=case["steps"]) for s, md in zip(state["systems"], state["md"])]
        got = [srv.result(i) for i in ids]
        return {"x": [r[0].astype(out) for r in got], "v": [r[1].astype(out) for r in got]}
    eng, s = state["engine"], state["system"]
    if case["call"] == "force":
        eng.upload_state(state["x"])
        eng.mklist_cell()
        f, e, v = eng.calforce()
        return {"force": f.astype(out), "energies": _energies(e).astype(out),
                "virials": np.concatenate([np.atleast_1d(v[k]) for k in sorted(v)]).astype(out)}
    if case["call"] == "ewk":
        eng.upload_state(state["x"])
        r = eng.ewaldkp_hf(case["kmax"])
        return {k: r[k] for k in ("force", "pot_atm", "viri_atm", "pot_virit_coul")} | {
            "pot": np.array([r["pot_ewk"], r["pot_ewk_cc"]]), "nwave": r["nwave"]}
    ens, n = case.get("ens", "nve"), case["steps"]
    if ens != "nve":
        eng.set_chain(abi.chain_init(s.box))
    step = {"nve": eng.moldyn_nve, "nhc": eng.moldyn_nhc, "mtk": eng.moldyn_mtk}[ens]
    eng.upload_state(state["x"], state["v"], s.box)
    got = {}
    if case["call"] == "host":
        x, v = state["x_out"], state["v_out"]
        for k in range(n + 1):
            e = step(k, k, state["md"])
            eng.download_state(x, v)
            if k < n:
                eng.upload_state(x, v)
    elif case["call"] == "hf":
        e, rec = eng.moldyn_hf(0, n, state["md"], cap=n)
        got["flux"] = rec.astype(out)
    else:
        e = step(0, n, state["md"])
    x, v, box = eng.download_state(state["x_out"], state["v_out"])
    return {"x": x.astype(out), "v": v.astype(out), "box": box.astype(out), "energies": _energies(e).astype(out), **got}


def _energies(e):
    return np.array([e[k] for k in abi.ENERGY_NAMES])


# ---- what a pass cannot do without ---------------------------------------------------
def work(case):
    if case["call"] == "serve":
        every = [_step_work(s, s.params) for s in _replicas(case, 0)]
        n = case["steps"] + 1
        return {"bytes": sum(n * 96.0 * a + 96.0 * a for a, _ in every), "flops": sum(n * f for _, f in every)}
    s = _system(case, 0)
    natom, flops = _step_work(s, s.params)
    if case["call"] == "ewk":
        # half the wave sphere: a wave and its opposite have conjugate phases
        waves = 2.0 / 3.0 * math.pi * case["kmax"] ** 3
        return {"bytes": 24.0 * natom + 104.0 * natom, "flops": 50.0 * natom * waves}
    if case["call"] == "force":
        return {"bytes": 48.0 * natom, "flops": flops}
    n = case["steps"] + 1
    host = 96.0 * natom * (n if case["call"] == "host" else 1)
    if case["call"] == "hf":   # per pair: two energies, two z-resolved virials
        flops += 60.0 * _pairs(s, s.params)
    return {"bytes": 96.0 * natom * n + host, "flops": flops * n}


def _pairs(s, p):
    volume = float(np.prod(s.box)) if not s.regions else s.natom / 0.1   # a slab: its own density, not the box's
    return 0.5 * s.natom * (s.natom / volume) * 4.0 / 3.0 * math.pi * max(p["rcut"], p["rrcut"]) ** 3


def _step_work(s, p):
    """(atoms, flops of one force evaluation): 61 per pair, the two transforms, the B-spline spread and gather, ~150 per
    bonded term."""
    k3 = float(p["nfft1"] * p["nfft2"] * p["nfft3"])
    terms = len(s.bonds) + len(s.angles) + 2 * len(s.tors) + 2 * len(s.torsrb)
    return s.natom, (61.0 * _pairs(s, p) + 5.0 * k3 * math.log2(k3) + 10.0 * s.natom * p["pme_order"] ** 3 +
                     150.0 * terms)


# ---- the same in 64 bits, in plain torch ---------------------------------------------
def exact(case, seed):
    """Same layout as run(); None where no short calculation gives it: virials (the engine's split by term), dynamics with
    a barostat, of a slab with random forces or of flexible molecules' heat flux, and what takes minutes at this size."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["call"] == "serve":
        if case["steps"] * case["high"] > 4_000_000:
            return None
        got = [_dynamics(_Exact(s, dev), _md(s, "nve", ""), "nve", case["steps"]) for s in _replicas(case, seed)]
        return {"x": [g["x"] for g in got], "v": [g["v"] for g in got]}
    s = _system(case, seed)
    if case["call"] == "ewk":
        return _ewald_waves(s, case["kmax"], dev)
    if case["call"] == "force":
        if s.natom > 100_000:
            return None
        f, e = _Exact(s, dev).force(torch.tensor(s.atmcor, device=dev))
        return {"force": f.cpu().numpy(), "energies": e, "virials": None}
    if case.get("ens") == "mtk" or case["kind"] == "slab" or s.natom ** 2 * case["steps"] > 1e10:
        return None
    flux = None
    if case["call"] == "hf":
        if case["kind"] != "water":
            return None
        flux = _heat_flux(case, s)["regions"]
    return _dynamics(_Exact(s, dev), _md(s, case.get("ens", "nve"), case["kind"]), case.get("ens", "nve"), case["steps"],
                     flux)


class _Exact:
    """Energy and force of a system: Lennard-Jones, Ewald (real space, smooth particle mesh, excluded pairs) and bonded
    terms, every pair of atoms by itself, derivatives of the mesh and bonded energies by autograd."""

    def __init__(self, s, dev):
        t = lambda a, d=torch.float64: torch.as_tensor(np.asarray(a), device=dev, dtype=d)  # noqa: E731
        i = lambda a: t(a, torch.int64)  # noqa: E731
        self.s, self.p, self.dev = s, s.params, dev
        self.box, self.q, self.m, self.type = t(s.box), t(s.atmchrg), t(s.atmmass), i(s.atmindex) - 1
        self.r2min, self.well = t(s.vdw_radij) ** 2, t(s.vdw_welij)
        rows = np.diff(s.index_excl)
        ei, ej = np.repeat(np.arange(s.natom), rows), s.list_excl[: rows.sum()] - 1
        self.ei, self.ej = i(ei[ej >= 0]), i(ej[ej >= 0])
        self.bonds, self.bk, self.br = i(s.bonds), t(s.bond_k), t(s.bond_r0)
        self.angles, self.ak, self.at = i(s.angles), t(s.angl_k), t(s.angl_t0)
        self.tors, self.tb, self.td = i(s.tors), t(s.tors_barhig), t(s.tors_divfac)
        self.rb, self.rc = i(s.torsrb), t(s.torsrb_c)
        self.p14 = torch.cat([self.tors[:, [0, 3]], self.rb[:, [0, 3]]])
        self.f14 = torch.cat([t(s.tors_delc), t(s.torsrb_delc)]), torch.cat([t(s.tors_dvdw), t(s.torsrb_dvdw)])
        self.first = i(s.molept_list[s.molept_index[:-1]])
        self.mol = i(np.repeat(np.arange(s.nmole), np.diff(s.molept_index)))
        self.cut = float(s.params["rrcut"]), float(s.params["rcut"])
        self._mesh()
        # the k-th constraint of every group at once: groups share no atom
        idx = [s.const_list[a:b] for a, b in zip(s.const_index[:-1], s.const_index[1:])]
        most = max((len(g) for g in idx), default=0)
        cols = [np.array([g[k] for g in idx if len(g) > k]) for k in range(most)]
        self.cons = [(i(s.const_ij[c, 0]), i(s.const_ij[c, 1]), t(s.const_d[c])) for c in cols]

    def image(self, d):
        return d - self.box * torch.round(d / self.box)

    def rows(self):
        n = self.s.natom
        step = max(1, 24_000_000 // n)
        for a in range(0, n, step):
            b = min(n, a + step)
            pick = (self.ei >= a) & (self.ei < b), (self.ej >= a) & (self.ej < b)
            out = torch.ones(b - a, n, dtype=torch.bool, device=self.dev)
            out[self.ei[pick[0]] - a, self.ej[pick[0]]] = False
            out[self.ej[pick[1]] - a, self.ei[pick[1]]] = False
            out[torch.arange(b - a), torch.arange(a, b)] = False
            yield a, b, out

    def lj(self, r2, a, b):
        ti, tj = self.type[a], self.type[b]
        s6 = (self.r2min[ti, tj] / r2) ** 3
        e = self.well[ti, tj]
        return e * (s6 * s6 - 2.0 * s6), 12.0 * e * (s6 * s6 - s6) / r2

    def pairs(self, x):
        """Force, LJ and real-space Coulomb energy of the pairs inside the cutoffs."""
        alpha, f = float(self.p["alpha"]), torch.zeros_like(x)
        ev = ec = 0.0
        for a, b, ok in self.rows():
            d = self.image(x[a:b, None] - x[None])
            r2 = (d * d).sum(-1)
            i, j = (ok & (r2 <= max(self.cut) ** 2)).nonzero(as_tuple=True)
            d, r2, i = d[i, j], r2[i, j], i + a
            r = r2.sqrt()
            qq = self.q[i] * self.q[j] * (r <= self.cut[0])
            erfc = torch.erfc(alpha * r)
            ec += 0.5 * float((qq * erfc / r).sum())
            fs = qq * (erfc / r + 2.0 * alpha / math.sqrt(math.pi) * torch.exp(-alpha * alpha * r2)) / r2
            e, g = self.lj(r2, i, j)
            near = r2 <= self.cut[1] ** 2
            ev += 0.5 * float((e * near).sum())
            f.index_add_(0, i, (fs + g * near)[:, None] * d)
        return f, ev, ec

    def _mesh(self):
        p, pi = self.p, math.pi
        k, order, alpha = (p["nfft1"], p["nfft2"], p["nfft3"]), p["pme_order"], float(p["alpha"])
        h, mod = [], []
        for d in range(3):
            w = torch.zeros(k[d], dtype=torch.float64, device=self.dev)
            w[1: order + 1] = torch.stack(self.spline(torch.zeros((), dtype=torch.float64, device=self.dev), order))
            m = torch.fft.fft(w).abs() ** 2
            for c in range(1, k[d] - 1):
                if m[c] < 1e-7:
                    m[c] = 0.5 * (m[c - 1] + m[c + 1])
            mod.append(m)
            n = torch.arange(k[d], device=self.dev, dtype=torch.float64)
            h.append(torch.where(n < (k[d] + 1) // 2, n, n - k[d]) / self.box[d])
        msq = h[0][:, None, None] ** 2 + h[1][None, :, None] ** 2 + h[2][None, None, :] ** 2
        m = [0.5 * k[d] / float(self.box[d]) for d in range(3)]
        top = m[0]
        top = m[1] if m[1] < m[0] else top
        top = m[2] if m[2] < m[1] else top
        keep = (msq > 0) & (msq <= (0.9 * top) ** 2)
        den = pi * float(self.box.prod()) * mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, :] * msq
        self.influence = torch.where(keep, torch.exp(-pi * pi / alpha ** 2 * msq) / den.clamp_min(1e-300), 0.0 * msq)

    @staticmethod
    def spline(w, order):
        """Cardinal B-spline weights of a fractional offset w, lowest grid point first."""
        m = [1.0 - w, w]
        for n in range(3, order + 1):
            up = [(1.0 - w) * m[0] / (n - 1)]
            up += [((w + (n - 1 - c)) * m[c - 1] + (c + 1 - w) * m[c]) / (n - 1) for c in range(1, n - 1)]
            m = up + [w * m[-1] / (n - 1)]
        return m

    def mesh(self, x):
        p = self.p
        k, order = (p["nfft1"], p["nfft2"], p["nfft3"]), p["pme_order"]
        grid = torch.zeros(k[0] * k[1] * k[2], dtype=torch.float64, device=self.dev)
        w, at = [], []
        for d in range(3):
            u = x[:, d] / self.box[d]
            u = (u - torch.floor(u)) * k[d]
            base = u.detach().floor()
            w.append(self.spline(u - base, order))
            at.append([(base.long() - order + 1 + c) % k[d] for c in range(order)])
        for a in range(order):
            for b in range(order):
                for c in range(order):
                    grid = grid.index_add(0, (at[0][a] * k[1] + at[1][b]) * k[2] + at[2][c],
                                          self.q * w[0][a] * w[1][b] * w[2][c])
        spec = torch.fft.fftn(grid.view(k))
        return 0.5 * (self.influence * (spec.real ** 2 + spec.imag ** 2)).sum()

    def dihedral(self, x, t):
        a, b, c = (self.image(x[t[:, 1]] - x[t[:, 0]]), self.image(x[t[:, 1]] - x[t[:, 2]]),
                   self.image(x[t[:, 3]] - x[t[:, 2]]))
        n1, n2 = torch.linalg.cross(a, b), torch.linalg.cross(b, c)
        return (n1 * n2).sum(-1) / (n1.norm(dim=-1) * n2.norm(dim=-1))

    def terms(self, x):
        zero = x.sum() * 0.0
        alpha = float(self.p["alpha"])
        r = self.image(x[self.ei] - x[self.ej]).norm(dim=-1)
        e = {"excluded": -(self.q[self.ei] * self.q[self.ej] * torch.erf(alpha * r) / r).sum() if len(r) else zero}
        on = self.bk != 0
        r = self.image(x[self.bonds[on, 0]] - x[self.bonds[on, 1]]).norm(dim=-1)
        e["pot_bond"] = (self.bk[on] * (r - self.br[on]) ** 2).sum() + zero
        on = self.ak != 0
        i, j, k = self.angles[on].unbind(1)
        a, b = self.image(x[j] - x[i]), self.image(x[j] - x[k])
        th = torch.acos((a * b).sum(-1) / (a.norm(dim=-1) * b.norm(dim=-1)))
        e["pot_angl"] = (self.ak[on] * (th - self.at[on]) ** 2).sum() + zero
        c = self.dihedral(x, self.tors)   # every periodic torsion of these systems has period 3, phase 0
        e["pot_tors"] = (self.tb / self.td * (1.0 + 4.0 * c ** 3 - 3.0 * c)).sum() + zero
        c = -self.dihedral(x, self.rb)
        e["pot_torsrb"] = sum((self.rc[:, n] * c ** n).sum() for n in range(6)) + zero
        i, j = self.p14.unbind(1)
        r2 = (self.image(x[i] - x[j]) ** 2).sum(-1)
        e["pot_elc14"] = (self.q[i] * self.q[j] / r2.sqrt() / self.f14[0]).sum() + zero
        e["pot_vdw14"] = (self.lj(r2, i, j)[0] / self.f14[1]).sum() + zero
        e["pot_ewk"] = self.mesh(x)
        return e

    def force(self, x):
        f, ev, ec = self.pairs(x)
        x = x.detach().clone().requires_grad_(True)
        t = self.terms(x)
        f = f - torch.autograd.grad(sum(t.values()), x)[0]
        e = {k: float(v.detach()) for k, v in t.items()}
        e["pot_vdw"], e["pot_elc"], e["pot_mor"] = ev, ec + e["excluded"], 0.0
        alpha = float(self.p["alpha"])
        e["pot_ewc"] = -alpha / math.sqrt(math.pi) * float((self.q ** 2).sum())
        e["pot_ewnq"] = -0.5 * math.pi / (alpha ** 2 * float(self.box.prod())) * float(self.q.sum()) ** 2
        e["pot_nonbon"] = sum(e["pot_" + k] for k in ("vdw", "elc", "ewk", "ewc", "ewnq", "vdw14", "elc14"))
        e["pot_tot"] = e["pot_nonbon"] + sum(e["pot_" + k] for k in ("bond", "angl", "tors", "torsrb", "mor"))
        return f, _energies(e)

    def wrap(self, x):
        """Molecules whose first atom left the box are moved back as a whole."""
        a = x[self.first]
        return x + (((a < 0).double() - (a > self.box).double()) * self.box)[self.mol]

    def shake(self, x, old, v):
        for _ in range(300):
            worst = 0.0
            for i, j, d in self.cons:
                r, o = x[i] - x[j], old[i] - old[j]
                off = (r * r).sum(-1) - d * d
                g = (off / (2.0 * (r * o).sum(-1) * (1 / self.m[i] + 1 / self.m[j])))[:, None] * o
                for at, sign in ((i, -1.0), (j, 1.0)):
                    dx = sign * g / self.m[at][:, None]
                    x = x.index_add(0, at, dx)
                    v = v.index_add(0, at, dx / DT)
                worst = max(worst, float((off / (d * d)).abs().max()))
            if worst < 1e-13:
                break
        return x, v

    def project(self, x, v):
        for _ in range(300):
            worst = 0.0
            for i, j, d in self.cons:
                r = x[i] - x[j]
                rv = (r * (v[i] - v[j])).sum(-1)
                g = (rv / (d * d * (1 / self.m[i] + 1 / self.m[j])))[:, None] * r
                v = v.index_add(0, i, -g / self.m[i][:, None]).index_add(0, j, g / self.m[j][:, None])
                worst = max(worst, float((rv / (d * d)).abs().max()))
            if worst < 1e-12:
                break
        return v

    def flux(self, x, v, regions):
        """z heat flux of rigid water in slabs: kinetic, Coulomb and LJ transport, Coulomb and LJ collision."""
        kinds = {"elc": 7, "lj": 8}
        z, lz = x[:, 2], float(self.box[2])
        z = z + lz * ((z < 0).double() - (z >= lz).double())
        pot = {k: torch.zeros_like(z) for k in kinds}
        out = np.zeros((len(regions), abi.HF_NCOL))
        for a, b, ok in self.rows():
            d = self.image(x[a:b, None] - x[None])
            r2 = (d * d).sum(-1)
            i, j = (ok & (r2 <= max(self.cut) ** 2)).nonzero(as_tuple=True)
            d, r2, i = d[i, j], r2[i, j], i + a
            r = r2.sqrt()
            ee = self.q[i] * self.q[j] / r * (r <= self.cut[0])
            el, fl = self.lj(r2, i, j)
            near = r2 <= self.cut[1] ** 2
            fv = (d * v[i]).sum(-1)   # both orders of a pair come by: i's share only
            rz = z[i] - z[j]
            for name, e, fs in (("elc", ee, ee / r2), ("lj", el * near, fl * near)):
                pot[name].index_add_(0, i, 0.5 * e)
                for k, (z1, z2) in enumerate(regions):
                    part = (torch.maximum(z[i], z[j]).clamp(max=z2) - torch.minimum(z[i], z[j]).clamp(min=z1)).clamp(min=0)
                    part = part * torch.sign(rz) * (rz.abs() / lz < 0.5)
                    out[k, 8 + kinds[name]] += 0.5 * float((fs * fv * part).sum())
        kin = 0.5 * self.m * (v * v).sum(-1)
        for k, (z1, z2) in enumerate(regions):
            inside = (z1 <= z) & (z <= z2)
            out[k, 0] = float((kin * v[:, 2] * inside).sum())
            for name, c in kinds.items():
                out[k, c] = float((pot[name] * v[:, 2] * inside).sum())
            out[k] /= float(self.box[0] * self.box[1]) * (z2 - z1)
            out[k, 17] = out[k, :17].sum()
        return out


def _chain_half(c, md, kint, degfree):
    """Half a step of the Nose-Hoover chain (Yoshida-Suzuki factors)."""
    m, v, x = md.mchain, c["v"], c["x"]
    q, gkt = list(md.qmass), md.text

    def sweep(order, w4, w8):
        for i in order:
            g = (q[i - 1] * v[i - 1] ** 2 - gkt) / q[i]
            if i == m - 1:
                v[i] += g * w4
            else:
                e8 = math.exp(-w8 * v[i + 1])
                v[i] = v[i] * e8 * e8 + w4 * g * e8

    g0 = (kint - gkt * degfree) / q[0]
    for _ in range(md.next):
        for y in range(md.nyosh):
            w2 = md.yscoeff[y] * DT / md.next / 2.0
            w4, w8 = w2 / 2.0, w2 / 4.0
            sweep(range(m - 1, 0, -1), w4, w8)
            e8 = math.exp(-w8 * v[1])
            v[0] = v[0] * e8 * e8 + w4 * g0 * e8
            for i in range(m):
                x[i] += v[i] * w2
            v[0] = v[0] * e8 * e8 + w4 * g0 * e8
            sweep(range(1, m), w4, w8)


def _dynamics(ex, md, ens, steps, regions=None):
    """Steps 0..n of velocity Verlet with constraints, with a Nose-Hoover chain for "nhc"."""
    s = ex.s
    x, v = ex.wrap(torch.tensor(s.atmcor, device=ex.dev)), torch.tensor(s.atmvel, device=ex.dev)
    f, e = ex.force(x)
    chain = {"x": [0.0] * 8, "v": [0.0] * 8}
    kint = lambda v: float((ex.m * (v * v).sum(-1)).sum())  # noqa: E731
    rec = []
    for step in range(1, steps + 1):
        if step % 50 == 1:   # once per pair-list period
            x = ex.wrap(x)
        scale, kick = 1.0, 0.5 * DT
        if ens == "nhc":
            _chain_half(chain, md, kint(v), s.degfree_all)
            u = 0.25 * DT * chain["v"][0]
            scale = math.exp(-2.0 * u)
            u2 = u * u
            kick *= math.exp(-u) * (1 + u2 / 6 * (1 + u2 / 20 * (1 + u2 / 42 * (1 + u2 / 72))))
        v = v * scale + f / ex.m[:, None] * kick
        x, v = ex.shake(x + DT * v, x, v)
        f, e = ex.force(x)
        v = ex.project(x, v * scale + f / ex.m[:, None] * kick)
        if ens == "nhc":
            _chain_half(chain, md, kint(v), s.degfree_all)
        if regions:
            rec.append(ex.flux(x, v, regions))
    out = {"x": x.cpu().numpy(), "v": v.cpu().numpy(), "box": np.array(s.box), "energies": e}
    if regions:
        out["flux"] = np.stack(rec)
    return out


def _ewald_waves(s, kmax, dev):
    n = torch.arange(-kmax, kmax + 1, device=dev)
    w = torch.cartesian_prod(n, n, n)
    w = w[((w * w).sum(1) <= kmax * kmax) & ((w * w).sum(1) > 0)].double()
    t = lambda a: torch.tensor(a, device=dev, dtype=torch.float64)  # noqa: E731
    x, q, box, alpha = t(s.atmcor), t(s.atmchrg), t(s.box), float(s.params["alpha"])
    vol = float(box.prod())
    f, pot = torch.zeros_like(x), torch.zeros_like(q)
    vir, tot, energy = torch.zeros(len(q), 9, dtype=torch.float64, device=dev), torch.zeros(9, dtype=torch.float64, device=dev), 0.0
    for c in torch.split(w / box, 1024):
        k2 = (c * c).sum(1)
        a = torch.exp(-(math.pi / alpha) ** 2 * k2) / k2
        th = 2.0 * math.pi * (x @ c.T)
        sn, cs = torch.sin(th), torch.cos(th)
        bs, bc = q @ sn, q @ cs
        shape = torch.eye(3, device=dev, dtype=torch.float64).reshape(1, 9) - \
            ((2.0 / k2 + 2.0 * (math.pi / alpha) ** 2)[:, None, None] * c[:, :, None] * c[:, None, :]).reshape(-1, 9)
        pa = 0.5 / math.pi / vol * a * (sn * bs + cs * bc) * q[:, None]
        pw = 0.5 / math.pi / vol * a * (bs * bs + bc * bc)
        pot += pa.sum(1)
        vir += pa @ shape
        tot += pw @ shape
        energy += float(pw.sum())
        f += 2.0 / vol * q[:, None] * ((a * (bc * sn - bs * cs)) @ c)
    pot -= alpha / math.sqrt(math.pi) * q * q
    return {"force": f.cpu().numpy(), "pot_atm": pot.cpu().numpy(), "viri_atm": vir.view(-1, 3, 3).cpu().numpy(),
            "pot_virit_coul": tot.view(3, 3).cpu().numpy(), "pot": np.array([energy, 0.0]), "nwave": len(w) + 1}
