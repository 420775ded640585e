"""The work that users of disco_b200 have it do, as cases that can be timed and compared.

A disk case is what a simulation program does between two looks at its state:
`steps` RK2 timesteps of a batch (disco_batch_run, or with loop "host" the
reference's own main loop, dt = getmindt; timestep(dt), between an upload and
a download of the whole state, as the drop-in into a Disco host runs it), then
the download of what a checkpoint holds of every cell: the primitives, the
face fluxes of constrained transport, the cell positions, into pinned host
buffers that the program keeps.  The mixed form holds its primitives in FP32 and
moves its mesh with them: its program keeps the primitives, as FP32.  A c2p case is calc_prim's loop alone: the GRMHD
cons->prim solve of n cells on device arrays.

    listed()            the cases, as dicts
    draw(rng)           one more of the same ranges
    prepare(case, seed) the batch or solver with its inputs, on the GPU
    run(state)          one pass
    work(case)          the bytes and operations of a pass
    exact(case, seed)   2D hydro and c2p: the pass's results in 64-bit torch
"""
import ctypes as C
import math
import os

import numpy as np
import torch

import disco_b200 as db
from disco_b200 import gr as dgr
from disco_b200.workloads import ragged_specs, write_par

R_IN, R_OUT = 0.5, 3.0                  # the 2D Keplerian disk's radii (c0_kepler2d)


def listed():
    return [
        # the smallest disk in use (the smallest of the ragged batch): every
        # launch is short, the step is a chain of launches
        dict(name="hydro nr32", kind="hydro", nr=32, ndisk=1, prec="fp64", steps=10, loop="graph"),
        # the reference's plain model: one 2D Keplerian disk of 128 annuli
        dict(name="hydro nr128", kind="hydro", nr=128, ndisk=1, prec="fp64", steps=10, loop="graph"),
        # the drop-in's use: a host program uploads its domain, steps it with
        # its own dt loop and takes the domain back
        dict(name="hydro dropin nr201", kind="hydro", nr=201, ndisk=1, prec="fp64", steps=5, loop="host"),
        # a parameter study: 64 disks of 32 to 256 annuli and Mach 10 to 40 in one batch
        dict(name="ragged64", kind="ragged", nr=256, ndisk=64, prec="fp64", steps=10, loop="graph"),
        # the same in the FP32 form, for long runs
        dict(name="ragged64 mixed", kind="ragged", nr=256, ndisk=64, prec="mixed", steps=20, loop="graph"),
        # 3D MHD shearing disk, HLLD, zero-gradient boundaries, B through the fluxes
        dict(name="mhd 64x64", kind="mhd", nr=64, nz=64, ct=0, prec="fp64", steps=5),
        # the same in the FP32 form on a small, odd grid (a test run)
        dict(name="mhd 37x21 mixed", kind="mhd", nr=37, nz=21, ct=0, prec="mixed", steps=5),
        # the shearing disk with constrained transport
        dict(name="mhd ct 64x64", kind="mhd", nr=64, nz=64, ct=1, prec="fp64", steps=5),
        # a quarter of the large circumbinary disk (128 layers), in its FP32 form
        dict(name="binary nz32 mixed", kind="binary", nr=384, nz=32, prec="mixed", steps=10),
        # a thin slab of it in FP64, for comparing against the FP32 form
        dict(name="binary nz4", kind="binary", nr=384, nz=4, prec="fp64", steps=3),
        # GRMHD torus, Kerr-Schild spin 0.9, a slice of 16 layers
        dict(name="grtorus 192x16", kind="grtorus", nr=192, nz=16, prec="fp64", steps=3),
        # the GRMHD cons->prim solve alone, as a host code's calc_prim calls it
        dict(name="c2p 946k", kind="c2p", n=946176, nextra=10, eps=1e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hydro", "hydro", "ragged", "mhd", "mhd", "binary", "grtorus", "c2p"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "hydro":
        loop = rng.choice(["graph", "graph", "host"])
        return dict(kind=kind, nr=_log_int(rng, 32, 256), ndisk=1, prec=prec,
                    steps=10 if loop == "graph" else 5, loop=loop)
    if kind == "ragged":
        return dict(kind=kind, nr=_log_int(rng, 64, 256), ndisk=_log_int(rng, 3, 64), prec=prec,
                    steps=10, loop="graph")
    if kind == "mhd":
        return dict(kind=kind, nr=_log_int(rng, 20, 80), nz=_log_int(rng, 6, 64), ct=rng.choice([0, 1]),
                    prec=prec, steps=5)
    if kind == "binary":
        return dict(kind=kind, nr=384, nz=_log_int(rng, 2, 20), prec=prec, steps=4)
    if kind == "grtorus":
        return dict(kind=kind, nr=_log_int(rng, 48, 192), nz=_log_int(rng, 6, 24), prec="fp64", steps=3)
    return dict(kind=kind, n=_log_int(rng, 20000, 4000000) | 1, nextra=rng.choice([0, 10, 10]),
                eps=rng.choice([1e-3, 1e-3, 0.3]))


# ---- prepare ---------------------------------------------------------------

def _disk(base, opt, over):
    par = write_par(over, base=base)
    try:
        return db.Disk.from_files(par, os.path.join(db.TEMPLATES, opt + ".in"))
    finally:
        os.unlink(par)


def _disks(case, seed):
    s = 1 + seed % 1000000007            # in.par's Init_Par0, an int
    kind = case["kind"]
    if kind == "hydro":
        return [_disk("c0_kepler2d", "c0_kepler2d", {"Num_R": case["nr"], "Init_Par0": s})]
    if kind == "ragged":
        # the batch's seeded sizes and Mach numbers, the sizes scaled to nr
        return [_disk("c0_kepler2d", "c0_kepler2d",
                      {"Num_R": max(32, nr * case["nr"] // 256), "Mach_Number": repr(mach), "Init_Par0": s + i})
                for i, (nr, mach, _) in enumerate(ragged_specs(case["ndisk"]))]
    if kind == "mhd":
        return [_disk("c1_mhd3d", "c1_mhd3d", {"Num_R": case["nr"], "Num_Z": case["nz"],
                                               "Constrained_Transport": case["ct"], "Init_Par0": s})]
    if kind == "binary":
        nz = case["nz"]                  # the mid-plane slab of nz of the 128 layers
        return [_disk("c4_binary3d", "c4_binary3d", {"Num_R": case["nr"], "Num_Z": nz, "Z_Min": -0.5 * nz / 128,
                                                     "Z_Max": 0.5 * nz / 128, "Init_Par0": s})]
    nz = case["nz"]                      # the torus's mid-plane slice of nz of 96 layers
    return [_disk("c3_grtorus", "c3_grtorus_kerr",
                  {"Num_R": case["nr"], "Num_Z": nz, "Z_Min": -20.0 * nz / 96, "Z_Max": 20.0 * nz / 96,
                   "aspect": 0.75, "Metric_Par3": 0.9, "Init_Par0": s})]


def _pinned(*shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=True)
    return t, t.numpy()


def _prepare_c2p(case, seed):
    """Cells of the torus grid: the previous prims and the conserved variables of a later state."""
    solver = dgr.GR(metric="kerr", a=0.9, tol=1e-10, nextra=case["nextra"], max_iter=30)
    np_ = 462
    nz = max(1, case["n"] // (np_ * 64))
    nr = -(-case["n"] // (np_ * nz))
    x = solver.grid(nr, nz, np_, 1.5, 50.0, -20.0, 20.0)[:, :case["n"]].contiguous()
    before = solver.torus(x, dgr.torus_defaults(a=0.9, seed=1 + seed))
    later = solver.perturb(before, 7 + seed, case["eps"])
    return dict(solver=solver, x=x, before=before, later=later, cons=solver.prim2cons(later, x),
                prim=torch.empty_like(before))


def prepare(case, seed):
    if case["kind"] == "c2p":
        return dict(case=case, **_prepare_c2p(case, seed))
    disks = _disks(case, seed)
    batch = db.Batch(disks, precision=db.PREC_MIXED if case["prec"] == "mixed" else db.PREC_FP64)
    n, q = batch.ncell, batch.q
    st = dict(case=case, batch=batch, n=n)
    st["tprim"], st["prim"] = _pinned(n, q)
    _, st["piph"] = _pinned(n)
    if batch.ct:
        _, st["Phi"] = _pinned(n, batch.num_faces)
    if case["prec"] == "mixed":
        st["prim32"] = torch.empty((n, q), dtype=torch.float32)
    if case.get("loop") == "host":
        out = {"prim": st["prim"], "piph": st["piph"]}
        for k, shape in (("cons", (n, q)), ("dphi", (n,)), ("wiph", (n,))):
            out[k] = _pinned(*shape)[1]
        first = batch.get_cells(out=out)
        st["out"] = out
        st["host"] = {}
        for k, v in first.items():
            st["host"][k] = _pinned(*v.shape)[1]
            st["host"][k][...] = v
        st["real"] = np.concatenate([d.real for d in disks]).astype(np.int32)
    return st


# ---- run -------------------------------------------------------------------

def _ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double)) if a is not None else None


def _download(st):
    """What a checkpoint holds of the cells, through the C ABI (NULL skips an array)."""
    s = db.library().disco_batch_get_cells(st["batch"].h, _ptr(st["prim"]), None, _ptr(st["piph"]), None, None,
                                           _ptr(st.get("Phi")))
    if s != db.OK:
        raise db.DiscoError(s, "disco_batch_get_cells")


def run(state):
    case = state["case"]
    if case["kind"] == "c2p":
        state["prim"].copy_(state["before"])            # the warm start; solved in place
        state["solver"].cons2prim(state["cons"], state["x"], state["prim"], stats=False)
        return {"prim": state["prim"]}
    batch = state["batch"]
    mixed = case["prec"] == "mixed"
    if case.get("loop") == "host":
        h = state["host"]
        batch.set_cells(h["prim"], h["cons"], h["piph"], h["dphi"], h["wiph"], state["real"])
        for _ in range(case["steps"]):
            batch.timestep(batch.mindt())
        out = dict(batch.get_cells(out=state["out"]))
    else:
        batch.run(case["steps"])
        _download(state)
        out = {"prim": state["prim"], "piph": state["piph"]}
        if "Phi" in state:
            out["Phi"] = state["Phi"]
    if mixed:
        state["prim32"].copy_(state["tprim"])           # FP32 values: nothing is lost
        return {"prim": state["prim32"]}
    return out


# ---- work ------------------------------------------------------------------

def _cells(case):
    """Cells of a case (ghost annuli left out): the reference's setupGrid counts."""
    kind = case["kind"]
    if kind in ("hydro", "ragged"):
        nrs = [case["nr"]] if kind == "hydro" else [max(32, nr * case["nr"] // 256)
                                                    for nr, _, _ in ragged_specs(case["ndisk"])]
        return sum(nr * int(2 * math.pi / (1.0 - (R_OUT / R_IN) ** (-1.0 / nr))) for nr in nrs)
    r0, r1, aspect, log = {"mhd": (1.0, 4.0, 1.34, False), "binary": (0.5, 10.0, 1.66, False),
                           "grtorus": (1.5, 50.0, 0.75, True)}[kind]
    nr = case["nr"]
    n = 0
    for j in range(nr):
        if log:
            n += max(4, int(2 * math.pi / (aspect * (1.0 - (r1 / r0) ** (-1.0 / nr)))))
        else:
            dr = (r1 - r0) / nr
            n += max(4, int(2 * math.pi / (aspect * dr / (r0 + (j + 1) * dr))))
    return n * case["nz"]


def work(case):
    if case["kind"] == "c2p":
        # cons, x and the warm start read, the solution written; about 60
        # operations per Newton iteration, two and the tail of them, 400 around them
        return {"bytes": case["n"] * 8.0 * (9 + 3 + 9 + 9), "flops": case["n"] * (400.0 + 60.0 * (2 + case["nextra"]))}
    n = _cells(case)
    q = 6 if case["kind"] in ("hydro", "ragged") else 9
    ct = 5 if case["kind"] == "binary" or case.get("ct") else 0
    w = 4 if case["prec"] == "mixed" else 8
    # a step reads and writes the cell's state once: cons, the prims, the face
    # fluxes, piph, dphi, wiph (and the FP32 form's carry of cons)
    step = 2 * (8 * q + w * q + 8 * ct + 24 + (4 * q if w == 4 else 0))
    out = 8 * (q + 1 + ct)
    if case.get("loop") == "host":
        out = 2 * 8 * (2 * q + 3)
    ops = {"hydro": 1500, "ragged": 1500, "mhd": 5000, "binary": 6500, "grtorus": 9000}[case["kind"]]
    return {"bytes": float(n) * (case["steps"] * step + out), "flops": float(n) * case["steps"] * ops}


# ---- exact -----------------------------------------------------------------

def exact(case, seed):
    """2D hydro disks: the same steps of the same disk (Euler, HLLC, PLM, RK2, the sun's
    gravity, fixed boundaries, a mesh that moves with the gas) in 64-bit torch.  c2p: the
    prims whose conserved variables the solve was given.  The 3D MHD and GRMHD steps have
    no such value here."""
    if case["kind"] == "c2p":
        return {"prim": _prepare_c2p(case, seed)["later"]}
    if case["kind"] not in ("hydro", "ragged"):
        return None
    disks = _disks(case, seed)
    batch = db.Batch(disks, precision=db.PREC_MIXED if case["prec"] == "mixed" else db.PREC_FP64)
    first = batch.get_cells()
    batch.close()
    sim = Hydro2D([(d.params, d.Nr, d.Ng, d.Np, d.r_jph, d.z_kph) for d in disks], first,
                  "cuda" if torch.cuda.is_available() else "cpu")
    for _ in range(case["steps"]):
        sim.step()
    if case["prec"] == "mixed":
        return {"prim": sim.prim}
    out = {"prim": sim.prim, "piph": sim.piph}
    if case.get("loop") == "host":
        out.update(cons=sim.cons, dphi=sim.dphi, wiph=sim.wiph)
    return out


class Hydro2D:
    """The 2D Keplerian hydro disks of a batch, stepped in 64-bit torch: all annuli of all
    disks in one set of flat arrays, the faces between neighbouring annuli by sorting their
    cells' edges in phi, the sums over a cell's faces by index_add."""

    RHO, PPP, URR, UPP, UZZ, PAS = range(6)

    def __init__(self, disks, first, device):
        def t(a, dt=torch.float64):
            return torch.as_tensor(np.asarray(a), device=device).to(dt)
        par = disks[0][0]
        self.dev = device
        self.gam, self.theta, self.cfl, self.tau = par.Adiabatic_Index, par.PLM, par.CFL, 2 * math.pi
        ann_np, rp, rm, adisk, aj, mach, real, edge = [], [], [], [], [], [], [], []
        trA, dxL, dxR, tr_r, tflux = [], [], [], [], []
        na = 0
        for d, (p, Nr, Ng, Np, rj, zk) in enumerate(disks):
            cen = 2.0 * (rj[1:]**2 + rj[1:] * rj[:-1] + rj[:-1]**2) / (3.0 * (rj[1:] + rj[:-1]))
            for j in range(Nr):
                ann_np.append(int(Np[j])); rp.append(rj[j + 1]); rm.append(rj[j]); adisk.append(d); aj.append(j)
                mach.append(p.Disk_Mach); real.append(Ng[0] <= j < Nr - Ng[1])
                edge.append(-1 if j == 0 else 1 if j == Nr - 1 else 0)
                if j < Nr - 1:
                    trA.append(na + j); dxL.append(rj[j + 1] - cen[j]); dxR.append(cen[j + 1] - rj[j + 1])
                    tr_r.append(rj[j + 1]); tflux.append(Ng[0] - 1 <= j < Nr - Ng[1])
            na += Nr
        dz = float(disks[0][5][1] - disks[0][5][0])
        self.dz = dz
        npt = t(ann_np, torch.int64)
        self.off = torch.cumsum(npt, 0) - npt
        self.n = int(npt.sum())
        self.ann = torch.repeat_interleave(torch.arange(na, device=device), npt)
        loc = torch.arange(self.n, device=device) - self.off[self.ann]
        self.prev = self.off[self.ann] + (loc - 1) % npt[self.ann]
        self.next = self.off[self.ann] + (loc + 1) % npt[self.ann]
        per = lambda a: t(a)[self.ann]
        self.rp, self.rm, self.mach = per(rp), per(rm), per(mach)
        self.r = 2.0 * (self.rp**2 + self.rp * self.rm + self.rm**2) / (3.0 * (self.rp + self.rm))
        self.real = t(real, torch.bool)[self.ann]
        self.edge = t(edge, torch.int64)[self.ann]
        self.disk = t(adisk, torch.int64)[self.ann]
        self.ndisk = len(disks)
        self.rmin, self.rmax = par.rmin, par.rmax
        # faces: entry e of track k is an edge of annulus A (side 0) or A + 1 (side 1)
        A = t(trA, torch.int64)
        nA, nB = npt[A], npt[A + 1]
        cnt = nA + nB
        nt = len(trA)
        self.tr = torch.repeat_interleave(torch.arange(nt, device=device), cnt)
        self.toff = (torch.cumsum(cnt, 0) - cnt)[self.tr]
        e = torch.arange(self.tr.numel(), device=device) - self.toff
        self.tn, self.tnA, self.tnB = cnt[self.tr], nA[self.tr], nB[self.tr]
        self.side = (e >= self.tnA).to(torch.int64)
        self.pos = torch.where(self.side == 0, self.off[A][self.tr] + e, self.off[A + 1][self.tr] + e - self.tnA)
        self.baseA, self.baseB = self.off[A][self.tr], self.off[A + 1][self.tr]
        self.local = e
        trk = lambda a: t(a)[self.tr]
        self.dxL, self.dxR, self.fr = trk(dxL), trk(dxR), trk(tr_r)
        self.fflux = t(tflux, torch.bool)[self.tr]
        self.prim, self.cons = t(first["prim"]), t(first["cons"])
        self.piph, self.dphi, self.wiph = t(first["piph"]), t(first["dphi"]), t(first["wiph"])
        self.dt = self.mindt()

    def wrap(self, x):                      # into [0, 2 pi]
        x = torch.where(x < 0, x + self.tau, x)
        return torch.where(x > self.tau, x - self.tau, x)

    def signed(self, x):                    # into [-pi, pi]
        x = torch.where(x < -0.5 * self.tau, x + self.tau, x)
        return torch.where(x > 0.5 * self.tau, x - self.tau, x)

    def om(self, r):                        # the energy's frame: Keplerian
        return r**-1.5

    def mindt(self):
        w = 0.5 * (self.wiph[self.prev] + self.wiph)
        p = self.prim
        cs = torch.sqrt(self.gam * p[:, self.PPP] / p[:, self.RHO])
        dtr = (self.rp - self.rm) / (cs + p[:, self.URR].abs())
        dtp = 0.5 * (self.rp + self.rm) * self.dphi / (cs + ((p[:, self.UPP] - w) * self.r).abs())
        dtz = self.dz / (cs + p[:, self.UZZ].abs())
        dt = torch.minimum(torch.minimum(dtr, dtp), dtz)
        dt = torch.where(self.real, dt, torch.full_like(dt, 1e300))
        out = torch.full((self.ndisk,), 1e300, dtype=torch.float64, device=self.dev)
        return self.cfl * out.scatter_reduce(0, self.disk, dt, "amin")

    def faces(self):
        key, o1 = torch.sort(self.piph, stable=True)
        order = o1[torch.sort(self.ann[o1], stable=True)[1]]   # by annulus, then phi
        cell = order[self.pos]
        phi = self.piph[cell]
        s1 = torch.sort(phi, stable=True)[1]
        s = s1[torch.sort(self.tr[s1], stable=True)[1]]
        isA = 1 - self.side[s]
        c = torch.cumsum(isA, 0) - isA
        ka = c - c[self.toff]
        kb = self.local - ka
        self.L = order[self.baseA + ka % self.tnA]
        self.R = order[self.baseB + kb % self.tnB]
        xp = phi[s]
        before = torch.where(self.local == 0, self.toff + self.tn - 1, torch.arange(s.numel(), device=self.dev) - 1)
        self.fdp = self.wrap(xp - xp[before])
        self.fphi = self.wrap(xp - 0.5 * self.fdp)
        self.fdA = self.fr * self.fdp * self.dz
        mid = self.piph - 0.5 * self.dphi
        self.dpL = self.signed(self.fphi - mid[self.L])
        self.dpR = self.signed(mid[self.R] - self.fphi)

    def slopes(self):
        p, d = self.prim, self.dphi[:, None]
        pL, pR, dL, dR = p[self.prev], p[self.next], d[self.prev], d[self.next]
        a = self.theta * (p - pL) / (0.5 * (d + dL))
        b = (pR - pL) / (0.5 * (dL + dR) + d)
        c = self.theta * (pR - p) / (0.5 * (dR + d))
        m = torch.where(a * b < 0, torch.zeros_like(a), a)
        m = torch.where(b.abs() < m.abs(), b, m)
        m = torch.where(b * c < 0, torch.zeros_like(a), m)
        self.gp = torch.where(c.abs() < m.abs(), c, m)
        L, R = self.L, self.R
        S = (p[R] - self.dpR[:, None] * self.gp[R] - p[L] - self.dpL[:, None] * self.gp[L]) / (self.dxL + self.dxR)[:, None]
        g = torch.zeros_like(p)
        g.index_add_(0, L, S * self.fdA[:, None])
        g.index_add_(0, R, S * self.fdA[:, None])
        dAp, dAm = self.rp * self.dphi * self.dz, self.rm * self.dphi * self.dz
        tot = torch.where(self.edge < 0, dAp, torch.where(self.edge > 0, dAm, dAp + dAm))
        g = g / tot[:, None]
        least = torch.full_like(p, math.inf)
        away = torch.zeros_like(p)
        for X in (L, R):
            ix = X[:, None].expand(-1, p.shape[1])
            least.scatter_reduce_(0, ix, (self.theta * S).abs(), "amin")
            away.scatter_reduce_(0, ix, (S * g[X] < 0).to(p.dtype), "amax")
        g = torch.sign(g) * torch.minimum(g.abs(), least)
        self.gr = torch.where(away > 0, torch.zeros_like(g), g)

    def flux(self, p, r, n):                # n: 0 phi, 1 r
        rho, P, vr, vp, vz = p[:, 0], p[:, 1], p[:, 2], p[:, 3] * r, p[:, 4]
        vn = vr if n == 1 else vp
        off = self.om(r) * r
        v2 = vr**2 + (vp - off)**2 + vz**2
        e = P / (self.gam - 1)
        m = rho * vn
        F = torch.stack([m, (0.5 * rho * v2 + e + P) * vn - (P * off if n == 0 else 0), rho * vr * vn + (P if n == 1 else 0),
                         r * (rho * vp * vn + (P if n == 0 else 0)), rho * vz * vn, p[:, 5] * m], 1)
        return F

    def conserved(self, p, r):
        rho, P, vr, vp, vz = p[:, 0], p[:, 1], p[:, 2], p[:, 3] * r, p[:, 4]
        off = self.om(r) * r
        v2 = vr**2 + (vp - off)**2 + vz**2
        return torch.stack([rho, 0.5 * rho * v2 + P / (self.gam - 1), rho * vr, r * rho * vp, rho * vz, p[:, 5] * rho], 1)

    def star(self, p, r, n, Sk, Ss):
        rho, P, vr, vp, vz = p[:, 0], p[:, 1], p[:, 2], p[:, 3] * r, p[:, 4]
        vn = vr if n == 1 else vp
        off = self.om(r) * r
        v2 = vr**2 + (vp - off)**2 + vz**2
        Sso = Ss - (off if n == 0 else 0)
        rs = rho * (Sk - vn) / (Sk - Ss)
        Ps = P * (Ss - vn) / (Sk - Ss)
        Us = P / (self.gam - 1) * (Sk - vn) / (Sk - Ss)
        return torch.stack([rs, 0.5 * rs * v2 + Us + rs * Sso * (Ss - vn) + Ps,
                            rs * (vr + (Ss - vn if n == 1 else 0)), r * rs * (vp + (Ss - vn if n == 0 else 0)),
                            rs * vz, p[:, 5] * rs], 1)

    def hllc(self, pL, pR, r, n, w):
        """(F - w U*) of the face between states pL and pR that moves with w."""
        def parts(p):
            vn = p[:, 2] if n == 1 else p[:, 3] * r
            return p[:, 0], p[:, 1], vn, torch.sqrt(self.gam * p[:, 1] / p[:, 0])
        d1, P1, v1, c1 = parts(pL)
        d2, P2, v2, c2 = parts(pR)
        Ss = (P2 - P1 - d1 * v1 * c1 - d2 * v2 * c2) / (-d1 * c1 - d2 * c2)
        Sr = torch.maximum(c1 + v1, c2 + v2)
        Sl = torch.minimum(v1 - c1, v2 - c2)
        left = (w < Ss)[:, None]
        pk = torch.where(left, pL, pR)
        Sk = torch.where(left[:, 0], Sl, Sr)
        U, F = self.conserved(pk, r), self.flux(pk, r, n)
        Us = self.star(pk, r, n, Sk, Ss)
        out = ((w < Sl) | (w > Sr))[:, None]
        return torch.where(out, F - w[:, None] * U, F + Sk[:, None] * (Us - U) - w[:, None] * Us)

    def boundary(self):
        """The ghost annuli: the Keplerian disk at the cells' centres (Boundary/fixed.c)."""
        r = 0.5 * (self.rp + self.rm)
        cs = r**-0.5 / self.mach
        s = (self.piph - 0.5 * self.dphi) / self.tau
        p = torch.stack([torch.ones_like(r), cs * cs, torch.zeros_like(r), 1.0 / (r * torch.sqrt(r)), torch.zeros_like(r),
                         4.0 * s * (1.0 - s)], 1)
        self.prim = torch.where(self.real[:, None], self.prim, p)

    def primitive(self):
        dV = (0.5 * (self.rp + self.rm) * (self.rp - self.rm) * self.dphi * self.dz)
        c, r = self.cons, self.r
        rho = c[:, 0] / dV
        vr, vp, vz = c[:, 2] / dV / rho, c[:, 3] / dV / r / rho, c[:, 4] / dV / rho
        off = self.om(r) * r
        ke = 0.5 * rho * (vr**2 + (vp - off)**2 + vz**2)
        P = (self.gam - 1) * (c[:, 1] / dV - ke)
        p = torch.stack([rho, P, vr, vp / r, vz, c[:, 5] / c[:, 0]], 1)
        self.prim = torch.where(self.real[:, None], p, self.prim)
        self.boundary()

    def substep(self, dt, old, move):
        if old is not None:
            self.cons = 0.5 * self.cons + 0.5 * old
        self.faces()
        self.slopes()
        p = self.prim
        L, R = self.L, self.R
        fL = p[L] + self.gr[L] * self.dxL[:, None] + self.gp[L] * self.dpL[:, None]
        fR = p[R] - self.gr[R] * self.dxR[:, None] - self.gp[R] * self.dpR[:, None]
        G = self.hllc(fL, fR, self.fr, 1, torch.zeros_like(self.fr)) * (self.fdA * dt[self.disk[L]])[:, None]
        G = torch.where(self.fflux[:, None], G, torch.zeros_like(G))
        half = 0.5 * self.gp * self.dphi[:, None]
        Gp = self.hllc(p + half, (p - half)[self.next], self.r, 0, self.r * self.wiph)
        Gp = Gp * ((self.rp - self.rm) * self.dz * dt[self.disk])[:, None]
        new = self.cons - Gp + Gp[self.prev]
        new.index_add_(0, L, -G)
        new.index_add_(0, R, G)
        r, r1 = self.r, 0.5 * (self.rp + self.rm)
        dVdt = r1 * (self.rp - self.rm) * self.dphi * self.dz * dt[self.disk]
        rho, P, vr, omg = p[:, 0], p[:, 1], p[:, 2], p[:, 3]
        o, o1 = self.om(r), -1.5 * r**-2.5
        F = -1.0 / r**2                       # the sun
        new[:, 2] += dVdt * (rho * omg**2 * r + P / r1 + rho * F)
        new[:, 1] += dVdt * rho * (r * vr * o**2 - r**2 * (omg - o) * vr * o1 + F * vr)
        self.cons = torch.where(self.real[:, None], new, self.cons)
        if move:
            self.piph = self.wrap(self.piph + self.wiph * dt[self.disk])
            self.dphi = self.wrap(self.piph - self.piph[self.prev])
        self.primitive()

    def step(self):
        self.wiph = 0.5 * (self.prim[:, self.UPP] + self.prim[self.next, self.UPP])
        old = self.cons
        self.substep(self.dt, None, True)
        self.substep(0.5 * self.dt, old, False)
        self.dt = self.mindt()
