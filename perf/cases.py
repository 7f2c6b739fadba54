"""Performance cases of the MD engine: what a program that runs md_run's force and integration
path on the GPU calls, over the sizes and options it is used with.

Kinds
  snapshot  the potential energy and gradient of one set of coordinates (a frame of a
            trajectory): coordinates in, cell and pair lists built, dnergy
  md        `steps` MD steps with the state resident on the device, then the records of the
            run's output files: energies and temperature of every step, coordinates, velocities
  io        one MD step for a driver that keeps coordinates and velocities in host memory:
            state in, step, state out
  min       `steps` iterations of steepest descent from given coordinates

A mixed-precision run's records are single precision (REAL4 files of md_run's monitor), an
FP64 run's double precision (REAL8).  Systems are synthetic: a chain, rigid waters on a
jittered lattice at liquid density, ions; topologies depend on the sizes alone, coordinates,
orientations and velocities on the seed.
"""
import functools
import math
import random

import numpy as np
import torch

from j_presto_b200 import abi, engine, systems

RC = 12.0                       # CUTLEN; the list radius is RC + 1.5
EEKCAL = 332.06378
KGAS, CONVCV = 8.31451, 4.184e-4
METHODS = {"MICR": abi.JP_METHOD_MICR, "CANO": abi.JP_METHOD_CANO, "GE": abi.JP_METHOD_GE}
CAL15M = {"ZD": abi.JP_CAL15M_ZD, "ATOM": abi.JP_CAL15M_ATOM, "CMM": abi.JP_CAL15M_CMM}


def _case(name=None, kind="md", nres=0, nwat=0, ions=0, reps=1, nwat_hi=0, nres_hi=0, precision="mixed",
          method="CANO", cal15m="ZD", free=False, alsd=False, steps=20):
    c = dict(kind=kind, nres=nres, nwat=nwat, ions=ions, reps=reps, nwat_hi=nwat_hi, nres_hi=nres_hi,
             precision=precision, method=method, cal15m=cal15m, free=free, alsd=alsd, steps=steps)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest use: one frame of a small water box, where launches and copies weigh
        _case("snapshot_water_2k", "snapshot", nwat=700),
        # re-evaluating the frames of a production trajectory in double precision
        _case("snapshot_chain_23k_fp64", "snapshot", nres=40, nwat=7411, precision="fp64"),
        # a short peptide in a small box: the latency-bound end of plain canonical MD
        _case("md_peptide_2k", nres=6, nwat=700),
        # microcanonical MD of a small water box (energy conservation checks)
        _case("md_water_3k_micr", nwat=1000, method="MICR"),
        # an ordinary solvated protein-sized system, the common production run
        _case("md_chain_23k", nres=40, nwat=7411),
        # the same in double precision (reference runs)
        _case("md_chain_23k_fp64", nres=40, nwat=7411, precision="fp64"),
        # a large single system: salt water, a ragged number of molecules
        _case("md_salt_water_99k", nwat=33000, ions=100),
        # a driver that keeps the state itself and exchanges it every step
        _case("io_chain_23k", "io", nres=40, nwat=7411, steps=1),
        # a peptide in a water droplet without periodic boundary, Coulomb by cell multipoles
        _case("md_droplet_5k_cmm", nres=12, nwat=1500, cal15m="CMM", free=True),
        # relaxing a freshly built system before MD
        _case("min_chain_9k", "min", nres=16, nwat=2999),
        # multicanonical production: many replicas of uneven size in one context
        _case("mcmd_64_replicas_1m", nres=8, nres_hi=30, nwat=600, nwat_hi=9000, reps=64, method="GE"),
        # adaptive lambda dynamics: a batch of equal replicas with a scaled cluster
        _case("alsd_32_replicas_290k", nres=12, nwat=3000, reps=32, method="GE", alsd=True),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["snapshot", "md", "md", "md", "io", "min", "batch", "batch", "free"])
    fp64 = "fp64" if rng.random() < 0.3 else "mixed"
    if kind == "batch":
        alsd = rng.random() < 0.4
        lo = log_int(500, 2500)
        return _case(None, "md", nres=rng.choice([8, 12, 16]), nres_hi=0 if alsd else rng.choice([0, 20, 30]),
                     nwat=lo, nwat_hi=0 if alsd else lo + log_int(100, 5000), reps=log_int(2, 24), method="GE",
                     alsd=alsd)
    if kind == "free":
        return _case(None, "md", nres=rng.choice([8, 12]), nwat=log_int(600, 3000), free=True, precision=fp64,
                     cal15m=rng.choice(["ATOM", "CMM"]))
    nwat = log_int(700, 33000)
    nres = rng.choice([0, 6, 12, 16, 30])
    if kind == "min":
        return _case(None, kind, nres=nres, nwat=min(nwat, 9000), precision=fp64, steps=rng.randrange(11, 30))
    ions = rng.choice([0, 0, 17])
    if kind == "md":
        # a freshly built chain is equilibrated under a thermostat first
        method = rng.choice(["MICR", "CANO"]) if nres == 0 else "CANO"
        return _case(None, kind, nres=nres, nwat=nwat, ions=ions, precision=fp64, method=method,
                     steps=rng.choice([10, 17, 20]))
    return _case(None, kind, nres=nres, nwat=nwat, ions=ions, precision=fp64, steps=1)


# ---- systems ------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _solute(nres):
    """A chain with its neutralising ions (and two waters) in a box just large enough."""
    box = 28.0 if nres <= 16 else 36.0 if nres <= 30 else 45.0
    return box, systems.solvated_polymer(nres, 2, box=box, seed=100 + nres)


@functools.lru_cache(maxsize=256)
def _topology(nres, nwat, ions, free):
    """Topology of a chain of nres residues (0: none), nwat waters in all and `ions` pairs; the
    waters' lattice sites and the ions' places are fixed by the sizes."""
    rng = np.random.default_rng([nres, nwat, ions, int(free)])
    vol = (nwat + 4.0 * nres + 2.0 * ions) / systems.WATER_DENSITY
    sol_box, sol = _solute(nres) if nres else (0.0, None)
    if free:
        radius = (3.0 * vol / (4.0 * math.pi)) ** (1.0 / 3.0) + 1.5
        box = 2.0 * radius + 30.0
    else:
        box = max(vol ** (1.0 / 3.0), 28.0, sol_box)
    base = sol["cord"] + 0.5 * (box - sol_box) if nres else np.zeros((0, 3))
    if free and nres:   # the chain's box around the droplet's centre
        radius = max(radius, np.linalg.norm(base - 0.5 * box, axis=1).max() + 2.0)
        box = 2.0 * radius + 30.0
        base = sol["cord"] + 0.5 * (box - sol_box)
    nw = nwat - (2 if nres else 0)
    need = nw + 2 * ions
    n = int(math.ceil((need * (box ** 3 / vol if free else 1.0)) ** (1.0 / 3.0) - 1e-9))
    while True:
        a = box / n
        g = (np.arange(n) + 0.5) * a
        sites = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        if free:
            sites = sites[np.linalg.norm(sites - 0.5 * box, axis=1) < radius - 1.0]
        if nres and len(sites) >= need:
            ok = np.ones(len(sites), bool)
            for c0 in range(0, len(base), 32):   # chain atoms in runs: only the sites around a run
                run_, half = base[c0:c0 + 32], 0.5 * np.ptp(base[c0:c0 + 32], axis=0) + 2.8
                d = sites - 0.5 * (run_.max(0) + run_.min(0))
                near = np.flatnonzero((np.abs(d - box * np.round(d / box)) <= half).all(1))
                d = sites[near, None, :] - run_[None, :, :]
                d -= box * np.round(d / box)
                ok[near] &= (np.einsum("ijk,ijk->ij", d, d) > 2.8 ** 2).all(1)
            sites = sites[ok]
        if len(sites) >= need:
            break
        n += 1
    sites = sites[rng.permutation(np.sort(rng.choice(len(sites), size=need, replace=False)))]
    n0, nsolv = len(base), 3 * nw
    nt, c6, c12 = systems.lj_tables()
    ow = n0 + 3 * np.arange(nw, dtype=np.int32)
    types = np.array([systems.T_OW, systems.T_HW, systems.T_HW])
    ion_t = np.array([systems.T_NA, systems.T_CL] * ions, np.int64)
    mass_t = np.array([t[3] for t in systems.TYPES])
    typ = np.concatenate([sol["atype"] if nres else [], np.tile(types, nw), ion_t]).astype(np.int32)
    chg = np.concatenate([sol["charge"] if nres else [], np.tile([systems.Q_OW, systems.Q_HW, systems.Q_HW], nw),
                          [1.0, -1.0] * ions])
    mol = np.concatenate([sol["molecule"] if nres else [], np.full(nsolv, systems.MOL_WATER),
                          [systems.MOL_NA, systems.MOL_CL] * ions]).astype(np.int32)
    natom = n0 + nsolv + 2 * ions
    ex_n = np.concatenate([np.diff(sol["excl_ptr"]) if nres else [], np.full(nsolv, 2), np.zeros(2 * ions)])
    wex = (ow[:, None] + np.array([1, 2, 0, 2, 0, 1], np.int32)).reshape(-1)
    ex_idx = np.concatenate([sol["excl_idx"] if nres else np.zeros(0, np.int32), wex]).astype(np.int32)

    def cat(key, cols, rows, dtype=np.int32):
        first = np.asarray(sol[key], dtype) if nres else np.zeros((0,) + ((cols,) if cols > 1 else ()), dtype)
        return np.concatenate([first, np.asarray(rows, dtype)])

    empty = np.zeros(0)
    t = dict(
        natom=natom, box=np.full(3, box), mass=mass_t[typ], charge=chg, atype=typ, molecule=mol, ntype=nt, c6=c6,
        c12=c12, s14_vdw=np.full(nt, systems.S14_VDW), s14_ele=np.full(nt, systems.S14_ELE),
        excl_ptr=np.concatenate([[0], np.cumsum(ex_n)]).astype(np.int32), excl_idx=ex_idx,
        bond=cat("bond", 2, (ow[:, None] + np.array([0, 1, 0, 2])).reshape(-1, 2)),
        bond_k=cat("bond_k", 1, np.full(2 * nw, 553.0), float),
        bond_r0=cat("bond_r0", 1, np.full(2 * nw, systems.R_OH), float),
        angle=cat("angle", 3, ow[:, None] + np.array([1, 0, 2])), angle_k=cat("angle_k", 1, np.full(nw, 100.0), float),
        angle_theta0=cat("angle_theta0", 1, np.full(nw, systems.ANG_HOH), float),
        shake_n=cat("shake_n", 1, np.full(nw, 3)),
        shake_atoms=cat("shake_atoms", 4, np.concatenate([ow[:, None] + np.arange(3), np.full((nw, 1), -1)], 1)),
        shake_dist=cat("shake_dist", 6, np.tile([systems.R_OH, systems.R_HH, systems.R_OH, 0, 0, 0], (nw, 1)), float))
    for k in ("tors", "impr"):
        for f, cols in (("", 4), ("_k", 1), ("_nrot", 1), ("_phase", 1), ("_div", 1)) + ((("_nbf", 1),) if k == "tors" else ()):
            t[k + f] = sol[k + f] if nres else (np.zeros((0, 4), np.int32) if cols == 4 else empty)
    if nres:
        t["residues"] = sol["residues"]
    odd = np.floor(sites / a).sum(1).astype(int) % 2 == 1
    t["_place"] = (base, sites, odd, nw, min(0.15, 0.05 * a))
    return t


def _state(top, rng):
    """Coordinates and velocities at 300 K of one replica."""
    base, sites, odd, nw, jit = top["_place"]
    o = sites[:nw] + rng.uniform(-jit, jit, size=(nw, 3))
    # dipoles about z, the molecular planes of lattice neighbours across each other, both
    # tilted at random: no hydrogen starts on top of another molecule, as in a liquid
    bis = np.array([0.0, 0.0, 1.0]) + rng.normal(scale=0.15, size=(nw, 3))
    bis /= np.linalg.norm(bis, axis=1)[:, None]
    flat = np.where(odd[:nw, None], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]) + rng.normal(scale=0.15, size=(nw, 3))
    per = flat - (flat * bis).sum(1)[:, None] * bis
    per /= np.linalg.norm(per, axis=1)[:, None]
    h = 0.5 * systems.ANG_HOH
    w = np.stack([o, o + systems.R_OH * (math.cos(h) * bis + math.sin(h) * per),
                  o + systems.R_OH * (math.cos(h) * bis - math.sin(h) * per)], 1).reshape(-1, 3)
    ions = sites[nw:] + rng.uniform(-jit, jit, size=(len(sites) - nw, 3))
    x = np.concatenate([base + rng.uniform(-0.1, 0.1, size=3), w, ions])
    v = rng.normal(size=x.shape) * np.sqrt(8.31451e-7 * 300.0 / top["mass"])[:, None]
    v -= (top["mass"][:, None] * v).sum(0) / top["mass"].sum()
    return x, v


def _sizes(case):
    """(residues, waters) of every replica."""
    if not case["nwat_hi"]:
        return [(case["nres"], case["nwat"])] * case["reps"]
    r = random.Random(case["nwat"] * 1000003 + case["nwat_hi"])
    pool = sorted({case["nres"], (case["nres"] + max(case["nres"], case["nres_hi"])) // 2, max(case["nres"], case["nres_hi"])})
    return [(r.choice(pool), r.randint(case["nwat"], case["nwat_hi"])) for _ in range(case["reps"])]


def _tops(case, seed):
    tops = []
    for k, (nres, nwat) in enumerate(_sizes(case)):
        t = _topology(nres, nwat, case["ions"], case["free"])
        x, v = _state(t, np.random.default_rng([seed, k]))
        t = dict(t, cord=x, vel=v)
        if case["alsd"]:
            # walls steep enough to hold lambda on the weight's range
            t = systems.alsd_replica(t, seed=k, walls=20000.0)
        elif case["method"] == "GE":
            t["ge"] = systems.mcmd_weight(-1.0e7, 1.0e7)
        tops.append(t)
    return tops


def _params(case):
    kw = dict(precision=abi.JP_PREC_FP64 if case["precision"] == "fp64" else abi.JP_PREC_MIXED,
              method=METHODS[case["method"]], cal15m=CAL15M[case["cal15m"]],
              bounda=abi.JP_BOUND_NONE if case["free"] else abi.JP_BOUND_PBC)
    if case["kind"] == "min":
        kw["shake_method"] = abi.JP_SHAKE_NONE   # a relaxation moves the waters flexibly
    if case["alsd"]:
        kw.update(alsd=abi.JP_ALSD_LMD, lambda0=0.8, scale_terms=abi.JP_SCALE_TORS)
    return kw


# ---- the calls ----------------------------------------------------------------------------
def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    tops = _tops(case, seed)
    e = engine.Engine(tops, **_params(case))
    n = sum(e.natoms)
    s = dict(case=case, engine=e, x=_pinned(n, 3), v=_pinned(n, 3))
    s["x"][:] = np.concatenate([t["cord"] for t in tops])
    s["v"][:] = np.concatenate([t["vel"] for t in tops])
    if case["free"]:
        s["x0"], s["v0"] = s["x"].copy(), s["v"].copy()
    if case["kind"] in ("md", "io"):
        s["ene"] = _pinned(case["steps"], len(tops), abi.JP_MAXENE)
        s["temp"] = _pinned(case["steps"], len(tops))
    return s


def _record(case, **arrays):
    """The arrays as the run's records hold them."""
    return {k: a.astype(np.float32 if case["precision"] == "mixed" else np.float64) for k, a in arrays.items()}


def run(state):
    case, e = state["case"], state["engine"]
    if case["kind"] == "snapshot":
        e.set_state(0, cord=state["x"])
        e.rebuild()
        ene, grad = e.energy_grad(0)
        return _record(case, ene=ene, grad=grad)
    if case["kind"] == "min":
        e.set_state(0, cord=state["x"])
        e.rebuild()
        _, ene, rmsf, _ = e.minimize(max_loop=case["steps"], convgr=1e-3)
        x, _ = e.get_state(0)
        return _record(case, ene=ene, rmsf=rmsf, x=x)
    x, v, ene, temp = (state[k] for k in ("x", "v", "ene", "temp"))
    io = case["kind"] == "io"
    if case["free"]:   # a droplet's runs start from its restart file: it must not evaporate
        e.set_state(0, cord=state["x0"], vel=state["v0"])
        e.rebuild()
    e.step_io(x if io else None, v if io else None, x, v, ene, temp, nsteps=case["steps"])
    return _record(case, ene=ene, temp=temp, x=x, v=v)


def work(case):
    """Per force evaluation: 52 flops for every pair within the cut-off; per atom-step the
    position and velocity read and written, the force and the mass read (bytes)."""
    n = 0
    for nres, nwat in _sizes(case):
        n += 3 * nwat + 16 * nres + 2 * case["ions"]
    pairs = 0.5 * n * (3.0 * systems.WATER_DENSITY) * 4.0 / 3.0 * math.pi * RC ** 3
    evals = case["steps"] + 1 if case["kind"] == "min" else 1 if case["kind"] == "snapshot" else case["steps"]
    per_atom = 72 if case["kind"] == "snapshot" else 128
    return {"bytes": float(per_atom * n * evals + 48 * n), "flops": 52.0 * pairs * evals}


# ---- the same in 64 bits, plain torch -----------------------------------------------------
class _Exact:
    """One replica's potential energy, gradient and steps in 64 bits, over all pairs."""

    def __init__(self, top, case):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.top, self.case = top, case
        self.shk = case["kind"] != "min"

        def put(a, dtype=torch.float64):
            return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=self.dev)

        self.put = put
        self.n = top["natom"]
        self.box = None if case["free"] else put(top["box"])
        self.q = put(top["charge"] * math.sqrt(EEKCAL))
        self.typ = put(top["atype"], torch.int64)
        self.c6, self.c12 = put(top["c6"]), put(top["c12"])
        self.mass = put(top["mass"])
        zd = case["cal15m"] == "ZD"
        self.f = 1.0 / RC ** 3 if zd else 0.0
        self.b, self.z = 0.5 * self.f, 1.5 / RC if zd else 0.0
        ptr = np.asarray(top["excl_ptr"])
        self.ptr = ptr
        self.ex_i = np.repeat(np.arange(self.n), np.diff(ptr))
        self.ex_j = np.asarray(top["excl_idx"])
        once = self.ex_i < self.ex_j
        self.ei, self.ej = put(self.ex_i[once], torch.int64), put(self.ex_j[once], torch.int64)
        qe = self.q[self.ei] * self.q[self.ej]
        self.qe = qe
        self.dself = -0.5 * self.z * float((self.q ** 2).sum() + 2.0 * qe.sum())
        # constrained pairs drop their bonds and angles
        grp = np.full(self.n, -1)
        for k, (g, m) in enumerate(zip(top["shake_atoms"], top["shake_n"])):
            grp[g[:m]] = k
        tied = lambda a, b: self.shk & (grp[a] == grp[b]) & (grp[a] >= 0)  # noqa: E731
        bo, an = np.asarray(top["bond"]).reshape(-1, 2), np.asarray(top["angle"]).reshape(-1, 3)
        kb, ka = ~tied(bo[:, 0], bo[:, 1]), ~tied(an[:, 0], an[:, 2])
        self.bond = (put(bo[kb], torch.int64), put(top["bond_k"][kb]), put(top["bond_r0"][kb]))
        self.angle = (put(an[ka], torch.int64), put(top["angle_k"][ka]), put(top["angle_theta0"][ka]))
        self.dihe = [(put(np.asarray(top[k]).reshape(-1, 4), torch.int64), put(top[k + "_k"]), put(top[k + "_nrot"]),
                      put(top[k + "_phase"]), put(top[k + "_div"])) for k in ("tors", "impr")]
        to = np.asarray(top["tors"]).reshape(-1, 4)[np.asarray(top["tors_nbf"]) == 1]
        self.p14 = put(to[:, [0, 3]], torch.int64)
        # SHAKE groups by size: atoms, squared lengths
        sn, sa, sd = np.asarray(top["shake_n"]), np.asarray(top["shake_atoms"]), np.asarray(top["shake_dist"])
        self.groups = [(m, put(sa[sn == m, :m], torch.int64), put(sd[sn == m, :m * (m - 1) // 2] ** 2))
                       for m in (2, 3, 4) if self.shk and (sn == m).any()]
        # temperature sub-systems (molecule entries) and their degrees of freedom
        ids, sub = np.unique(top["molecule"], return_inverse=True)
        nfr = 3.0 * np.bincount(sub, minlength=len(ids))
        if self.shk:
            np.subtract.at(nfr, sub[sa[:, 0]], sn * (sn - 1) // 2)
        self.sub, self.nfr = put(sub, torch.int64), put(nfr)

    def image(self, d):
        return d if self.box is None else d - self.box * torch.round(d / self.box)

    def pairs(self, x):
        g = torch.zeros_like(x)
        e_el = e_lj = 0.0
        step = max(1, int(2e7) // self.n)
        for a in range(0, self.n, step):
            b = min(self.n, a + step)
            d = self.image(x[a:b, None, :] - x[None, :, :])
            r2 = (d * d).sum(-1)
            lo, hi = self.ptr[a], self.ptr[b]
            rows = torch.arange(b - a, device=self.dev)
            r2[rows, rows + a] = 1e30
            r2[self.put(self.ex_i[lo:hi] - a, torch.int64), self.put(self.ex_j[lo:hi], torch.int64)] = 1e30
            on = r2 <= RC * RC
            r2 = torch.where(on, r2, 1e30)
            ri = 1.0 / r2
            r = torch.sqrt(ri)
            r6 = ri * ri * ri
            qq = torch.where(on, self.q[a:b, None] * self.q[None, :], 0.0)
            v1 = self.c6[self.typ[a:b]][:, self.typ] * r6
            v2 = self.c12[self.typ[a:b]][:, self.typ] * r6 * r6
            e_el += 0.5 * float((qq * (r + torch.where(on, self.b * r2, 0.0) - self.z)).sum())
            e_lj += 0.5 * float((v2 - v1).sum())
            fs = qq * (ri * r - self.f) + (12.0 * v2 - 6.0 * v1) * ri
            g[a:b] = -(d * fs[..., None]).sum(1)
        return e_el, e_lj, g

    def bonded(self, x):
        """Energies by slot of the bonded and 1-4 terms and their gradient."""
        x = x.detach().requires_grad_(True)
        e = {}

        def vec(i, j):
            return self.image(x[i] - x[j])

        i, k, r0 = self.bond
        e[abi_slot("BOND")] = (k * (vec(i[:, 0], i[:, 1]).norm(dim=1) - r0) ** 2).sum()
        i, k, t0 = self.angle
        u, w = vec(i[:, 0], i[:, 1]), vec(i[:, 2], i[:, 1])
        th = torch.atan2(torch.linalg.cross(u, w, dim=1).norm(dim=1), (u * w).sum(1))
        e[abi_slot("ANGLE")] = (k * (th - t0) ** 2).sum()
        for (i, k, nr, ph, div), slot in zip(self.dihe, ("TORS", "IMPR")):
            b1, b2, b3 = vec(i[:, 1], i[:, 0]), vec(i[:, 2], i[:, 1]), vec(i[:, 3], i[:, 2])
            p, q = torch.linalg.cross(b1, b2, dim=1), torch.linalg.cross(b2, b3, dim=1)
            c = (p * q).sum(1) / (p.norm(dim=1) * q.norm(dim=1))
            cn = torch.where(nr == 1, c, torch.where(nr == 2, 2 * c * c - 1, 4 * c ** 3 - 3 * c))
            e[abi_slot(slot)] = (k / div * (1.0 + torch.cos(ph) * cn)).sum()
        i = self.p14
        r2 = (vec(i[:, 0], i[:, 1]) ** 2).sum(1)
        t1, t2 = self.typ[i[:, 0]], self.typ[i[:, 1]]
        e[abi_slot("VDW14")] = systems.S14_VDW * (self.c12[t1, t2] / r2 ** 6 - self.c6[t1, t2] / r2 ** 3).sum()
        e[abi_slot("ELE14")] = systems.S14_ELE * (self.q[i[:, 0]] * self.q[i[:, 1]] / torch.sqrt(r2)).sum()
        e["excess"] = (self.qe * self.b * (vec(self.ei, self.ej) ** 2).sum(1)).sum()
        tot = sum(e.values())
        g, = torch.autograd.grad(tot, x)
        return {k: float(v.detach()) for k, v in e.items()}, g

    def energy_grad(self, x):
        ene = np.zeros(abi.JP_MAXENE)
        el, lj, g = self.pairs(x)
        eb, gb = self.bonded(x)
        ene[abi_slot("ELE15")] = el + eb.pop("excess") + self.dself
        ene[abi_slot("VDW15")] = lj
        for k, v in eb.items():
            ene[k] = v
        ene[0] = ene[1:].sum()
        return ene, g + gb

    def shake(self, x1, x0):
        """x1 constrained against x0: exact for two atoms, Newton with md_run's stop otherwise."""
        x1 = x1.clone()
        for m, atoms, len2 in self.groups:
            p = [(0, 1), (1, 2), (2, 0), (3, 0), (2, 3), (1, 3)][:m * (m - 1) // 2]
            im = 1.0 / self.mass[atoms]
            r1, r0 = x1[atoms], x0[atoms]
            d1 = torch.stack([self.image(r1[:, a] - r1[:, b]) for a, b in p], 1)
            d2 = torch.stack([self.image(r0[:, a] - r0[:, b]) for a, b in p], 1)
            inc = torch.zeros((m, len(p)), dtype=torch.float64, device=self.dev)
            for k, (a, b) in enumerate(p):
                inc[a, k], inc[b, k] = 1.0, -1.0
            cg = torch.einsum("aq,ga,ai->gqi", inc, im, inc)
            lam = torch.zeros_like(len2)
            if m == 2:
                a2, b2 = (cg[:, 0, 0] ** 2) * (d2 ** 2).sum((1, 2)), cg[:, 0, 0] * (d1 * d2).sum((1, 2))
                c2 = (d1 ** 2).sum((1, 2)) - len2[:, 0]
                lam[:, 0] = -(b2 - torch.sqrt(b2 * b2 - a2 * c2)) / a2
            else:
                wk = d1.clone()
                for _ in range(1000):
                    res = len2 - (wk ** 2).sum(-1)
                    todo = (res.abs() >= 1e-6 * len2).any(1)
                    if not bool(todo.any()):
                        break
                    mat = 2.0 * cg * torch.einsum("gqk,gik->gqi", wk, d2)
                    dl = torch.linalg.solve(mat, res)
                    lam += torch.where(todo[:, None], dl, 0.0)
                    wk = d1 + torch.einsum("gqi,gik->gqk", cg, d2 * lam[..., None])
            x1[atoms] = r1 + im[..., None] * torch.einsum("aq,gqk->gak", inc, d2 * lam[..., None])
        return x1

    def temps(self, v):
        ek = torch.zeros_like(self.nfr).index_add_(0, self.sub, self.mass * (v * v).sum(1))
        return ek * 1.0e7 / (KGAS * self.nfr), float(ek.sum() * 1.0e7 / (KGAS * self.nfr.sum()))

    def scale(self, ene):
        if self.case["method"] != "GE":
            return 1.0
        ge = self.top["ge"]
        rt = (ene[0] - ge["celw"]) / (ge["ceup"] - ge["celw"])
        return KGAS / 4.184e3 * ge["tempce"] * float(np.polynomial.polynomial.polyval(rt, ge["coef"][0]))

    def step(self, x, v, dt=2.0, t0=300.0):
        ene, g = self.energy_grad(x)
        acc = -CONVCV * self.scale(ene) * g / self.mass[:, None]
        if self.case["method"] == "MICR":
            x1 = self.shake(x + dt * (v + dt * acc), x)
            vn = (x1 - x) / dt
            return ene, self.temps(0.5 * (v + vn))[1], x1, vn
        chi = torch.sqrt(t0 / self.temps(v + 0.5 * dt * acc)[0])[self.sub][:, None]
        xb = x + dt * ((2.0 * chi - 1.0) * v + chi * dt * acc)
        con = torch.zeros_like(x)
        for it in range(1, 4):
            x1 = self.shake(xb, x)
            vn = (x1 - x) / dt
            t, tot = self.temps(0.5 * (v + vn))
            if it == 3 or float((t - t0).abs().max()) < 1e-3 * t0:
                return ene, tot, x1, vn
            con = con + (x1 - xb) / dt ** 2
            chi = torch.sqrt(t0 / self.temps(v + 0.5 * dt * (acc + con))[0])[self.sub][:, None]
            xb = x + dt * (chi * dt * (acc + con) + (2.0 * chi - 1.0) * v)


def abi_slot(name):
    """Index of an energy term in eneval."""
    return ["TOTAL", "BOND", "ANGLE", "TORS", "IMPR", "VDW14", "ELE14", "VDW15", "ELE15"].index(name)


def exact(case, seed):
    if case["alsd"] or case["cal15m"] == "CMM":
        return None   # class-weighted and multipole forces: no short plain form
    tops = _tops(case, seed)
    evals = case["steps"] + 1 if case["kind"] == "min" else 1 if case["kind"] == "snapshot" else case["steps"]
    if evals * sum(float(t["natom"]) ** 2 for t in tops) > 6.0e10:
        return None   # all pairs of that many atoms and steps take too long
    out = []
    for t in tops:
        E = _Exact(t, case)
        x, v = E.put(t["cord"]), E.put(t["vel"])
        if case["kind"] == "snapshot":
            ene, g = E.energy_grad(x)
            return dict(ene=ene, grad=g.cpu().numpy())
        if case["kind"] == "min":
            ene, g = E.energy_grad(x)
            stp, best = 0.01 * math.sqrt(E.n), ene[0]
            for _ in range(case["steps"]):
                x = x - stp / float(g.norm()) * g
                ene, g = E.energy_grad(x)
                stp, best = stp * (1.2 if ene[0] < best else 0.6), ene[0]
            rmsf = float(g.norm()) / math.sqrt(E.n)
            return dict(ene=ene[None], rmsf=np.array([rmsf]), x=x.cpu().numpy())
        rows, temps = [], []
        for _ in range(case["steps"]):
            ene, temp, x, v = E.step(x, v)
            rows.append(ene)
            temps.append(temp)
        out.append((np.stack(rows), np.array(temps), x.cpu().numpy(), v.cpu().numpy()))
    return dict(ene=np.stack([o[0] for o in out], 1), temp=np.stack([o[1] for o in out], 1),
                x=np.concatenate([o[2] for o in out]), v=np.concatenate([o[3] for o in out]))
