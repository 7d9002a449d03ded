"""The work that programs built on this library give it, as cases to time.

Five kinds of pass, each through the entry points a program calls:

  md        a stretch of the device-resident r-RESPA driver (Engine.md_run,
            then Engine.md_state): the library's main path.  Options: energy
            records, ORAC's thermostats, a non-equilibrium alchemical schedule
  batch     an interval of several systems advanced together (Batch.run with
            an energy record at its end, then every member's state): lambda
            windows and solute-scaled replicas
  resident  one evaluation of the M, L and H shells and of the reciprocal sum
            on coordinates that a caller keeps in device memory, forces only
            (orac_gpu_mts_forces_dev, orac_gpu_fft_pme_dev)
  host      what ORAC itself calls at a list-update step, with host arrays:
            lists, the three shells with energies and stress, fft_pme with
            its stress, and the intramolecular levels where there are any
  kspace    do_pmesh_kspace alone, on charges and a grid that the call brings

Systems are those of orac_b200.systems and the fixtures of tests/golden: rigid
waters, the bonded chain in water, the ligand in water, solvated chains of
2,000 to 81,000 atoms, and the protein-ligand system of the reference's own
test runs.  A seed moves every molecule as a whole by a few hundredths of an
Angstrom and draws new velocities at 300 K; the topology of a size is built
once per process.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(os.getcwd(), "orac-porting_b200")
if not os.path.isdir(PKG):
    PKG = os.path.join(ROOT, "orac-porting_b200")
GOLDEN = os.path.join(os.path.dirname(PKG), "tests", "golden")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
# parallel branches of a batch: as bench.py sets it for the same calls
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

from orac_b200 import oracio, systems, units  # noqa: E402
from orac_b200.engine import Batch, Engine  # noqa: E402

# the outer step (fs), L and M steps per outer and L step, list period, shell of
# the reciprocal sum, N1 and N0 substeps: the liquid water workload, the chains'
# with flexible bonds, and the reference's own test runs
WATER = dict(dt_h=4.0, lrespa=2, mrespa=4, nupdte=6, rshk="l", n1respa=1, n0respa=1)
PROTEIN = dict(dt_h=15.0, lrespa=5, mrespa=2, nupdte=6, rshk="l", n1respa=2, n0respa=2)


def listed():
    return [
        # the smallest system that the serving loop takes: latency and launches
        dict(name="md_chains_2k", kind="md", system="chains", natoms=2000, steps=12),
        # the headline workload: 3,000 rigid waters at liquid density
        dict(name="md_water_9k", kind="md", system="water", nwat=3000, steps=12),
        # a ligand in water under ORAC's thermostats, sampled every fourth step
        dict(name="md_ligand_nvt", kind="md", system="ligand", steps=12, every=4, thermostat=True),
        # the bonded 1,700-atom chain in water, spline order 5 on 64^3
        dict(name="md_chain_23k", kind="md", system="polymer", steps=10),
        # the reference's own test system and five-level schedule
        dict(name="md_protein", kind="md", system="protein", steps=3),
        # a walker of the reference's non-equilibrium work runs on that system
        dict(name="md_protein_work", kind="md", system="protein", steps=3, schedule=True),
        # the largest system that the serving loop takes
        dict(name="md_chains_81k", kind="md", system="chains", natoms=81000, steps=8),
        # lambda windows of the ligand, dU/dlambda at the interval's end
        dict(name="batch_windows_12", kind="batch", system="ligand", members=12, steps=12),
        # solute-scaled replicas of uneven sizes between two exchange attempts
        dict(name="batch_replicas_6", kind="batch", system="chains", natoms=7000, members=6, steps=12),
        # forces on coordinates that stay on the device, a ragged size
        dict(name="resident_chains_31k", kind="resident", system="chains", natoms=31000),
        # ORAC's own call sequence at a list update, host arrays, protein
        dict(name="host_protein", kind="host", system="protein"),
        # a reciprocal sum alone, an uneven grid and a high order
        dict(name="kspace_60k", kind="kspace", ncharge=60000, n1=90, n2=80, n3=96, order=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "md", "batch", "batch", "resident", "host", "kspace"])
    if kind == "kspace":
        smooth = [n for n in range(27, 97) if systems._smooth(n)]
        return dict(kind=kind, ncharge=_log(rng, 700, 60000), n1=rng.choice(smooth), n2=rng.choice(smooth),
                    n3=rng.choice(smooth), order=rng.choice([4, 4, 5, 6, 7, 8]))
    if kind == "resident":
        return dict(kind=kind, system="chains", natoms=_log(rng, 2000, 60000))
    if kind == "host":
        return dict(kind=kind, system="chains", natoms=_log(rng, 2000, 20000))
    if kind == "batch":
        if rng.random() < 0.5:
            return dict(kind=kind, system="ligand", members=rng.randint(2, 12), steps=rng.randint(6, 12))
        return dict(kind=kind, system="chains", natoms=_log(rng, 3000, 10000), members=rng.randint(2, 6),
                    steps=rng.randint(6, 12))
    system = rng.choice(["chains", "chains", "water", "water", "ligand", "protein"])
    if system == "protein":
        c = dict(kind=kind, system=system, steps=rng.randint(1, 4), thermostat=rng.random() < 0.5)
        if not c["thermostat"] and rng.random() < 0.5:
            c["schedule"] = True
        return c
    if system == "ligand":
        return dict(kind=kind, system=system, steps=rng.randint(6, 12), thermostat=rng.random() < 0.5,
                    every=rng.choice([0, 2, 5]))
    if system == "water":
        return dict(kind=kind, system=system, nwat=_log(rng, 700, 12000), steps=rng.randint(6, 12),
                    thermostat=rng.random() < 0.3, every=rng.choice([0, 0, 3]))
    return dict(kind=kind, system=system, natoms=_log(rng, 2000, 60000), steps=rng.randint(5, 9),
                thermostat=rng.random() < 0.3)


# ------------------------------------------------------------------ systems


@functools.lru_cache(maxsize=None)
def _water(nwat):
    # the liquid workload's lattice spacing (44.7 A / 15 sites), any number of waters
    lattice = int(math.ceil(nwat ** (1.0 / 3.0) - 1e-9))
    box = 2.98 * lattice
    nc = systems.linked_cells_for(box, systems.Shells())
    n = systems.pme_grid_for(box)
    return systems.water_box(nwat=nwat, box=box, lattice=lattice, nfft=(n, n, n), ncell=(nc, nc, nc))


@functools.lru_cache(maxsize=None)
def _chains(natoms):
    return systems.solvated_chains(natoms, 7000 + natoms)


@functools.lru_cache(maxsize=None)
def _ligand():
    return systems.ligand_in_water()


@functools.lru_cache(maxsize=None)
def _polymer():
    return systems.polymer_in_water()


@functools.lru_cache(maxsize=None)
def _protein(schedule):
    tp, rst = oracio.split_arrays(dict(np.load(os.path.join(GOLDEN, "f0_fkbp12.npz"))))
    if schedule:
        sh = systems.Shells(rcutm=5.0, rtolm=0.3, rneim=0.5, rcutl=8.1, rtoll=0.3, rneil=0.5, rcuth=12.5, rtolh=0.3,
                            rneih=1.5)
        nfft = (48, 49, 48)
    else:
        sh = systems.Shells(rcutm=5.1, rtolm=0.3, rneim=0.4, rcutl=7.8, rtoll=0.3, rneil=0.5, rcuth=10.0, rtolh=0.3,
                            rneih=1.5)
        nfft = (48, 48, 48)
    s = oracio.system_from_orac(tp, rst, alphal=0.37, nfft=nfft, order=4, shells=sh, ncell=(18, 18, 18),
                                fudge=0.83333, lj_fudge=0.5, name="protein", rigid_hydrogen=True)
    if schedule:
        s.ss_alchemy = np.where(np.arange(s.ntap) < 52, -2, 1).astype(np.int32)
    return s


def _base(case, member=0):
    kind = case["system"]
    if kind == "water":
        return _water(case["nwat"])
    if kind == "ligand":
        return _ligand()
    if kind == "polymer":
        return _polymer()
    if kind == "protein":
        return _protein(bool(case.get("schedule")))
    # the members of a batch differ in size
    return _chains(case["natoms"] + 1111 * member)


def _system(case, seed, member=0):
    """The case's system with every molecule moved as a whole and new velocities."""
    s = _base(case, member).copy()
    rng = np.random.default_rng([seed, member, 77])
    shift = rng.normal(0.0, 0.02, (3, s.nprot))[:, s.atomp - 1]
    d = s.oc @ shift
    s.xp0, s.yp0, s.zp0 = s.xp0 + d[0], s.yp0 + d[1], s.zp0 + d[2]
    s.xyz_restart = None
    v = rng.standard_normal((3, s.ntap)) * np.sqrt(units.BOLTZ * 300.0 / units.UNITE / s.mass)
    v -= ((v * s.mass).sum(axis=1) / s.mass.sum())[:, None]
    s.vx, s.vy, s.vz = np.ascontiguousarray(v)
    return s


def _schedule(case):
    if case["system"] == "protein":
        return dict(PROTEIN, nupdte=4) if case.get("schedule") else PROTEIN
    return WATER


def _setup(e, case):
    w = _schedule(case)
    e.md_setup(w["dt_h"], w["lrespa"], w["mrespa"], w["nupdte"], w["rshk"], n1respa=w["n1respa"],
               n0respa=w["n0respa"])


# ------------------------------------------------------------------- passes


def prepare(case, seed):
    kind = case["kind"]
    if kind == "kspace":
        return _prepare_kspace(case, seed)
    if kind == "batch":
        engines = []
        for k in range(case["members"]):
            s = _system(case, seed, k)
            e = Engine(s)
            x = k / max(1, case["members"] - 1)
            if case["system"] == "ligand":
                # charges off over the first half of the windows, then the LJ
                e.set_alchemy(s.ss_alchemy, 0.5, 0.5)
                if x <= 0.5:
                    e.set_lambda(0.0, 0.0, 0.0, 2.0 * x, dlam=[0.0, 0.0, 0.0, 2.0])
                else:
                    e.set_lambda(0.0, 2.0 * x - 1.0, 0.0, 1.0, dlam=[0.0, 2.0, 0.0, 0.0])
            else:
                e.set_rem(s.rematom, 0, 0.6 ** x)
            _setup(e, case)
            engines.append(e)
        return dict(case=case, engines=engines, batch=Batch(engines))
    s = _system(case, seed)
    e = Engine(s)
    if kind == "host":
        return dict(case=case, engine=e)
    if kind == "resident":
        e.update_lists()
        dev = torch.device("cuda", 0)

        def up(*a):
            return torch.from_numpy(np.concatenate(a)).to(dev)

        st = torch.cuda.ExternalStream(e.lib.orac_gpu_get_stream(e.ctx), device=dev)
        return dict(case=case, engine=e, stream=st, xyz=up(e.xp0, e.yp0, e.zp0), grp=up(e.xpg, e.ypg, e.zpg),
                    mol=up(e.xpcm, e.ypcm, e.zpcm), f=torch.zeros(4, 3 * s.ntap, dtype=torch.float64, device=dev),
                    red=torch.zeros(16, dtype=torch.float64, device=dev))
    if case.get("thermostat"):
        e.set_thermostat(300.0, 20.0, 20.0, 20.0)
    if case.get("schedule"):
        t = np.load(os.path.join(GOLDEN, "ne_test4.npz"))["schedule"]
        e.set_alchemy(s.ss_alchemy, 0.5, 0.5, shifted=True, qshift=4.0, ljshift=0.35)
        e.set_lambda(0.0, 0.0, 0.0, 0.0)
        e.set_schedule(t[:, 0] * 1000.0, t[:, 1], t[:, 2], t[:, 3], t[:, 4])
    _setup(e, case)
    return dict(case=case, engine=e)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "md":
        e = state["engine"]
        rec = e.md_run(case["steps"], energy_every=case.get("every", 0))
        x, v = e.md_state()
        out = {"x": x, "v": v}
        if case.get("every", 0):
            out["records"] = rec
        if case.get("schedule"):
            out["work"] = e.md_work()[0]
        return out
    if kind == "batch":
        state["batch"].run(case["steps"], energy_every=case["steps"])
        out = {}
        for k, e in enumerate(state["engines"]):
            x, v = e.md_state()
            out["x%d" % k], out["v%d" % k] = x, v
            out["r%d" % k] = e.md_records(1)[0][0, 1:]
        return out
    if kind == "resident":
        e, f, red = state["engine"], state["f"], state["red"]
        with torch.cuda.stream(state["stream"]):
            f.zero_()
        xyz, grp, mol = state["xyz"].data_ptr(), state["grp"].data_ptr(), state["mol"].data_ptr()
        for k, sh in enumerate(b"mlh"):
            rc = e.lib.orac_gpu_mts_forces_dev(e.ctx, bytes([sh]), xyz, grp, mol, f[k].data_ptr(), None, None)
            if rc:
                raise RuntimeError(e.lib.orac_gpu_last_error(e.ctx).decode())
        rc = e.lib.orac_gpu_fft_pme_dev(e.ctx, xyz, mol, f[3].data_ptr(), red.data_ptr(), None)
        if rc:
            raise RuntimeError(e.lib.orac_gpu_last_error(e.ctx).decode())
        return {"m": f[0], "l": f[1], "h": f[2], "k": f[3], "sums": red}
    if kind == "host":
        e = state["engine"]
        e.update_lists()
        out = {}
        for sh in "mlh":
            F, en, st = e.mts_forces(sh)
            out[sh] = F
            out["e" + sh] = e.ue6(en)
            out["s" + sh] = st
        F, eer, st = e.fft_pme()
        out["k"], out["ek"], out["sk"] = F, eer, st
        if e.s.has_intra():
            out["n0"], out["e0"] = e.intra_n0()
            out["n1"], out["e1"] = e.intra_n1()
        return out
    return _run_kspace(state)


# ------------------------------------------------------ the reciprocal sum alone


def _kspace_inputs(case, seed):
    """Charges at liquid density in a box slightly off cubic, about 1 A a point."""
    rng = np.random.default_rng([seed, 5])
    n = case["ncharge"]
    edge = (n / 0.1) ** (1.0 / 3.0)
    nn = np.array([case["n1"], case["n2"], case["n3"]], float)
    edge = edge * (nn / nn.prod() ** (1.0 / 3.0)) ** 0.5
    x = rng.uniform(-0.5, 0.5, (3, n)) * edge[:, None]
    q = rng.normal(0.0, 0.4, n)
    q = (q - q.mean()) * units.charge_internal(1.0)
    return x, q, np.diag(1.0 / edge), float(edge.prod()), 0.35


def _prepare_kspace(case, seed):
    x, q, recip, vol, alpha = _kspace_inputs(case, seed)
    # a context of any topology carries the call; its own atoms are not used
    return dict(case=case, engine=Engine(systems.two_waters()), a=(x[0], x[1], x[2], q, recip, vol, alpha))


def _run_kspace(state):
    case = state["case"]
    F, eer, vir = state["engine"].do_pmesh_kspace(*state["a"], case["order"], (case["n1"], case["n2"], case["n3"]))
    return {"f": F, "eer": eer, "vir": vir}


# --------------------------------------------------------------- what a pass needs


def _evals(natoms, volume, r0, r1):
    """Atom pairs between two radii at the system's density."""
    return natoms * 0.5 * (natoms / volume) * 4.0 / 3.0 * math.pi * (r1 ** 3 - r0 ** 3)


def _size(case, member=0):
    """(atoms, volume, grid points, order, M/L/H radii) without building the system."""
    s = case["system"]
    if s == "protein":
        return 14900, 146000.0, 48 ** 3, 4, ((5.0, 8.1, 12.5) if case.get("schedule") else (5.1, 7.8, 10.0))
    r = (5.0, 7.5, 10.0)
    if s == "water":
        n = int(math.ceil(case["nwat"] ** (1.0 / 3.0) - 1e-9)) * 2.98
        return 3 * case["nwat"], n ** 3, systems.pme_grid_for(n) ** 3, 4, r
    if s == "ligand":
        return 8941, 44.7 ** 3, 48 ** 3, 4, r
    if s == "polymer":
        return 22700, 62.0 ** 3, 64 ** 3, 5, r
    n = case["natoms"] + 1111 * member
    box = (n / 0.095) ** (1.0 / 3.0)
    return n, box ** 3, systems.pme_grid_for(box) ** 3, 4, r


def _fft_flops(points):
    # real transform there and back, 2.5 n log2 n each
    return 5.0 * points * math.log2(points)


def _shell_flops(n, vol, r):
    """M and L pairs at 60 operations (LJ and Ewald), H pairs at 36."""
    return 60.0 * _evals(n, vol, 0.0, r[0]), 60.0 * _evals(n, vol, r[0], r[1]), 36.0 * _evals(n, vol, r[1], r[2])


def _pme_flops(n, points, order):
    return _fft_flops(points) + 10.0 * points + n * (2.0 * order ** 3 + 8.0 * order ** 3)


def work(case):
    kind = case["kind"]
    if kind == "kspace":
        n, pts = case["ncharge"], case["n1"] * case["n2"] * case["n3"]
        return {"bytes": 56.0 * n, "flops": _pme_flops(n, pts, case["order"])}
    b = f = 0.0
    for k in range(case.get("members", 1)):
        n, vol, pts, order, r = _size(case, k)
        m, l, h = _shell_flops(n, vol, r)
        pme = _pme_flops(n, pts, order)
        if kind in ("resident", "host"):
            b += 8.0 * (3 * n + n + n / 3 + 12 * n)
            f += m + l + h + pme
            continue
        w = _schedule(case)
        nl = w["lrespa"]
        nm = nl * w["mrespa"]
        ndrift = nm * w["n1respa"] * w["n0respa"]
        # the state read and written once, the constrained drifts at about 300 operations an atom
        b += 96.0 * n
        f += case["steps"] * (nm * m + nl * (l + pme) + h + ndrift * 300.0 * n)
    return {"bytes": b, "flops": f}


def tolerance(case):
    kind = case["kind"]
    if kind == "kspace":
        return {"rel": 1e-5, "max": 1e-4}
    if kind in ("resident", "host"):
        # forces 1e-5 relative RMS, as the parity tests ask
        return {"rel": 1e-5, "max": 2e-4}
    # forces that agree to about 1e-6, carried along by the equations of motion of
    # a liquid, which multiply a difference by up to 27 in 80 fs: against the same
    # steps with 64-bit forces the velocities were off by 1e-6 to 3e-6 after one
    # pass and by up to 8e-6 (largest 4e-4) after two of 48 fs
    return {"rel": 3e-5, "max": 2e-3}


# ------------------------------------------- the same numbers in 64-bit arithmetic

# A&S 7.1.26, the form that the path defines its erfc by (in the digits it is given in)
AS = (0.2548296, -0.28449674, 1.4214137, -1.453152, 1.0614054, 0.3275911)


def _erfc(x, exp):
    t = 1.0 / (1.0 + AS[5] * x)
    return ((((AS[4] * t + AS[3]) * t + AS[2]) * t + AS[1]) * t + AS[0]) * t * exp(-x * x)


def _exact_shells(s):
    """Per shell: forces (3, N), energies (LJ and Coulomb of slt, slv, mixed) and
    the molecular stress, from all group pairs in the shell's radii."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    t = functools.partial(torch.as_tensor, device=dev)
    co = t(np.asarray(s.co))
    sc = t(np.stack([s.xp0, s.yp0, s.zp0]).T.copy())
    gc = t(np.stack(s.group_centres()).T.copy())
    mc = t(np.stack(s.molecule_centres()).T.copy()) @ co.T
    first = t(s.grppt[:, 0].astype(np.int64) - 1)
    size = t((s.grppt[:, 1] - s.grppt[:, 0] + 1).astype(np.int64))
    mg = int(size.max())
    q, pm = t(s.charge), t(s.pmass)
    kind = t(s.nbtype.astype(np.int64) - 1)
    tab = t(np.asarray(s.type_table).astype(np.int64) - 1)
    c12, c6 = t(s.ecc12), t(s.ecc6)
    solute = t(s.ss_index.astype(np.int64))
    mol = t(s.atomp.astype(np.int64) - 1)
    n, g = s.ntap, s.ngrp
    # excluded pairs i < j as sorted keys
    keys, p = [], 0
    m = s.mapnl
    for i in range(n):
        keys.extend(i * n + int(j) - 1 for j in m[p + 1:p + 1 + m[p]])
        p += 1 + m[p]
    excl = t(np.sort(np.array(keys or [-1], dtype=np.int64)))
    sh = s.shells
    spec = {"m": (0.0, 0.0, sh.rcutm, sh.rtolm), "l": (sh.rcutm, sh.rtolm, sh.rcutl, sh.rtoll),
            "h": (sh.rcutl, sh.rtoll, sh.rcuth, sh.rtolh)}
    reach = max(v[2] + v[3] for v in spec.values())
    F = {k: torch.zeros(n, 3, dtype=torch.float64, device=dev) for k in spec}
    E = {k: torch.zeros(6, dtype=torch.float64, device=dev) for k in spec}
    S = {k: torch.zeros(3, 3, dtype=torch.float64, device=dev) for k in spec}
    step = max(1, 20_000_000 // g)
    for lo in range(0, g, step):
        hi = min(g, lo + step)
        d = gc[lo:hi, None] - gc[None]
        d = (d - 2.0 * torch.round(0.5 * d)) @ co.T
        near = ((d * d).sum(-1) < reach * reach) & (torch.arange(g, device=dev)[None] > torch.arange(lo, hi, device=dev)[:, None])
        gi, gj = near.nonzero(as_tuple=True)
        del d, near
        gi = gi + lo
        ds = gc[gi] - gc[gj]
        img = 2.0 * torch.round(0.5 * ds)
        R = (ds - img) @ co.T
        r2g = (R * R).sum(-1)
        for k, (ri, ti, ro, to) in spec.items():
            ri0, ro0 = ri + ti, ro + to
            rg = r2g.sqrt()
            out = (rg >= ro) & (rg < ro0)
            inn = (rg >= ri) & (rg < ri0)
            band = ((rg >= ri0) & (rg < ro)) | out | inn
            idx = band.nonzero(as_tuple=True)[0]
            rb, Rb, ob, ib = rg[idx], R[idx], out[idx], inn[idx]

            def sw(a, b, w):  # S = (b - 3 a + 2 R) (b - R)^2 / w^3 and its derivative
                u, v = (b - 3.0 * a + 2.0 * rb) / w ** 3, b - rb
                return u * v * v, -2.0 * u * v + 2.0 * v * v / w ** 3

            Sf, dS = torch.ones_like(rb), torch.zeros_like(rb)
            if to > 0:
                a, b = sw(ro, ro0, to)
                Sf, dS = torch.where(ob, a, Sf), torch.where(ob, b, dS)
            if ti > 0:
                a, b = sw(ri, ri0, ti)
                Sf, dS = torch.where(ib, 1.0 - a, Sf), torch.where(ib, -b, dS)
            skip = _erfc(s.alphal * ri, math.exp) < 10.0e-4
            I, J = gi[idx], gj[idx]
            V = torch.zeros_like(rb)
            fg = torch.zeros(len(idx), 3, dtype=torch.float64, device=dev)  # on the j group
            for a in range(mg):
                for b in range(mg):
                    on = ((size[I] > a) & (size[J] > b)).nonzero(as_tuple=True)[0]
                    ia, jb = first[I[on]] + a, first[J[on]] + b
                    key = torch.minimum(ia, jb) * n + torch.maximum(ia, jb)
                    pos = torch.searchsorted(excl, key).clamp_(max=len(excl) - 1)
                    lt = tab[kind[ia], kind[jb]]
                    lj = c6[lt] > 1e-12
                    ok = excl[pos] != key
                    if skip:
                        ok = ok & lj
                    on, ia, jb, lt, lj = on[ok], ia[ok], jb[ok], lt[ok], lj[ok]
                    x = ((sc[ia] - gc[I[on]]) - (sc[jb] - gc[J[on]])) @ co.T + Rb[on]
                    r2 = (x * x).sum(-1)
                    r = r2.sqrt()
                    r6 = torch.where(lj, 1.0 / r2 ** 3, torch.zeros_like(r2))
                    u = c12[lt] * r6 * r6 - c6[lt] * r6
                    f = (12.0 * c12[lt] * r6 * r6 - 6.0 * c6[lt] * r6) / r2
                    w = torch.zeros_like(u)
                    if not skip:
                        ar = s.alphal * r
                        qq = q[ia] * q[jb]
                        ec = _erfc(ar, torch.exp)
                        w = qq * ec / r
                        f = f + qq * (ec + 2.0 / math.sqrt(math.pi) * ar * torch.exp(-ar * ar)) / (r2 * r)
                    V.index_add_(0, on, u + w)
                    fv = (f * Sf[on])[:, None] * x
                    F[k].index_add_(0, ia, fv)
                    F[k].index_add_(0, jb, -fv)
                    fg.index_add_(0, on, -fv)
                    tt = solute[ia] + solute[jb] - 2  # 0 slt, 1 mixed, 2 slv
                    slot = torch.tensor([0, 2, 1], device=dev)[tt]
                    E[k].index_add_(0, slot, u * Sf[on])
                    E[k].index_add_(0, slot + 3, w * Sf[on])
            X = (-dS * V / rb)[:, None] * Rb
            for grp, sign in ((I, 1.0), (J, -1.0)):
                for a in range(mg):
                    on = (size[grp] > a).nonzero(as_tuple=True)[0]
                    at = first[grp[on]] + a
                    F[k].index_add_(0, at, sign * pm[at][:, None] * X[on])
            fg = fg - X
            # force on the j group times the arm from the i molecule to the j molecule's image
            S[k] += fg.T @ (img[idx] @ co.T)
    for k in spec:
        S[k] += F[k].T @ mc[mol]
    return ({k: F[k].T.contiguous() for k in spec}, E, S)


def _spline(w, order):
    """Cardinal B-spline weights of the points floor(u) - order + 1 + k, and their
    derivatives: M_n(x) = x/(n-1) M_{n-1}(x) + (n-x)/(n-1) M_{n-1}(x-1)."""
    x = w[:, None] + np.arange(order)[::-1][None]  # arguments of M_order, k ascending

    def m(n, x):
        if n == 2:
            return np.where((x >= 0) & (x <= 2), 1.0 - np.abs(x - 1.0), 0.0)
        return (x * m(n - 1, x) + (n - x) * m(n - 1, x - 1.0)) / (n - 1)

    return m(order, x), m(order - 1, x) - m(order - 1, x - 1.0)


def _moduli(n, order, twopi):
    pts = _spline(np.zeros(1), order)[0][0][::-1]  # M_order at order-1 .. 0
    arr = np.zeros(n)
    for j in range(min(order, n)):
        # the spline's values at its knots, in ascending order of the knot
        arr[(j + 1) % n] += pts[::-1][j]
    k = np.arange(n)[:, None] * np.arange(n)[None] * (twopi / n)
    mod = (np.cos(k) @ arr) ** 2 + (np.sin(k) @ arr) ** 2
    for i in range(n):
        if mod[i] < 1.0e-7:
            mod[i] = 0.5 * (mod[i - 1] + mod[(i + 1) % n])
    return mod


def _exact_kspace(x, q, recip, vol, alpha, order, nfft):
    """Energy and forces of the smooth particle-mesh sum in 64 bits.  The path's
    single-precision pi is kept: it is part of the sum's definition."""
    pi = float(np.float32(math.pi))
    n = len(q)
    w = recip.T @ x
    frac = (w - np.round(w) + 0.5) * np.array(nfft, float)[:, None]
    base = np.floor(frac).astype(np.int64)
    sp = [_spline(frac[d] - base[d], order) for d in range(3)]
    pts = [(base[d][:, None] - order + 1 + np.arange(order)[None]) % nfft[d] for d in range(3)]
    flat = (pts[0][:, :, None, None] * nfft[1] + pts[1][:, None, :, None]) * nfft[2] + pts[2][:, None, None, :]
    flat = flat.reshape(n, -1)

    def weights(a, b, c):
        return (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(n, -1)

    grid = np.bincount(flat.ravel(), weights=(weights(sp[0][0], sp[1][0], sp[2][0]) * q[:, None]).ravel(),
                       minlength=nfft[0] * nfft[1] * nfft[2]).reshape(nfft)
    hat = np.fft.fftn(grid)
    m = [np.where(np.arange(k) >= (k + 1) // 2, np.arange(k) - k, np.arange(k)).astype(float) for k in nfft]
    mm = np.stack(np.meshgrid(*m, indexing="ij"))
    h = np.einsum("ij,jabc->iabc", recip, mm)
    msq = (h * h).sum(0)
    b = [_moduli(k, order, 2.0 * pi) for k in nfft]
    den = pi * vol * b[0][:, None, None] * b[1][None, :, None] * b[2][None, None] * msq
    den[0, 0, 0] = 1.0
    g = np.exp(-(pi * pi / (alpha * alpha)) * msq) / den
    # the zero mode is left as it is in the convolution and out of the energy
    eer = 0.5 * float((g * np.abs(hat) ** 2).sum() - g[0, 0, 0] * abs(hat[0, 0, 0]) ** 2)
    phi = (np.fft.ifftn(hat * g).real * grid.size).ravel()[flat]
    grad = [-(phi * weights(*(sp[e][1] if e == d else sp[e][0] for e in range(3)))).sum(1) * nfft[d] * q
            for d in range(3)]
    return recip @ np.stack(grad), eer


def exact(case, seed):
    kind = case["kind"]
    if kind in ("md", "batch"):
        # trajectories: thousands of force evaluations, constraints and integrator
        return None
    if kind == "kspace":
        F, eer = _exact_kspace(*_kspace_inputs(case, seed), case["order"], (case["n1"], case["n2"], case["n3"]))
        return {"f": F, "eer": eer, "vir": None}
    s = _system(case, seed)
    F, E, S = _exact_shells(s)
    Fk, eer = _exact_kspace(s.cartesian(), s.charge, 0.5 * s.oc.T, s.volume, s.alphal, s.order, s.nfft)
    if kind == "resident":
        return {"m": F["m"].reshape(-1), "l": F["l"].reshape(-1), "h": F["h"].reshape(-1), "k": Fk.reshape(-1),
                "sums": None}
    out = {}
    for k in "mlh":
        e = E[k]
        # energies in the order LJ slt, slv, mixed, then Coulomb
        out[k], out["e" + k], out["s" + k] = F[k], e, S[k]
    out.update(k=Fk, ek=eer, sk=None)
    if s.has_intra():
        out.update(n0=None, e0=None, n1=None, e1=None)
    return out
