"""GPU kernels at the sizes where their tiles end, against the FP64 oracle:
the pair kernel's rows (one group pair to several passes, groups of up to 3,
4 and 8 atoms, half and whole warps a row, coordinates that are no number),
the list's rows (beyond the shared buffer, beyond the list's capacity), the
plane FFT (odd axes, one x line left over, planes too large for shared memory)
and the plan kept for calls that bring their own grid; and what a context
keeps from one topology to the next.  Tolerances as in the other parity tests: forces relative RMS <= 1e-5
(FP32 pair and spline arithmetic), energies 1e-6 of the terms' magnitudes.
"""
import numpy as np
import pytest

import oracle
from orac_b200 import systems

pytestmark = pytest.mark.gpu


def rel_rms(F, Fref):
    return float(np.sqrt(((F - Fref) ** 2).sum() / max((Fref ** 2).sum(), 1e-300)))


def small_shells():
    return systems.Shells(rcutm=3.5, rtolm=0.3, rneim=0.4, rcutl=5.5, rtoll=0.3, rneil=0.4, rcuth=8.0, rtolh=0.3,
                          rneih=0.6)


@pytest.mark.parametrize("nwat", [2, 3, 4, 17, 64, 65])
def test_rows_of_few_groups(nwat):
    """All-pairs lists of 2 to 65 groups: rows of no entry to several passes."""
    from orac_b200.engine import Engine

    s = systems.water_box(nwat=nwat, box=18.8, lattice=5, nfft=(20, 20, 20))
    s.ncell = None
    s.shells = small_shells()
    o, g = oracle.Oracle(s.copy()), Engine(s.copy())
    o.update_lists()
    g.update_lists()
    for sh in "mlh":
        Fr, uer, sr = o.shell(sh)
        Fg, en, sg = g.shell(sh)
        scale = np.abs(uer).sum() + 1e-300
        # relative RMS; a shell without pairs has no forces on either side
        assert np.sqrt(((Fg - Fr) ** 2).sum()) <= 1e-5 * np.sqrt((Fr ** 2).sum()), sh
        assert np.abs(g.ue6(en) - uer).max() <= 1e-6 * scale
        assert np.linalg.norm(sg - sr) <= 1e-5 * max(np.linalg.norm(sr), 1e-12)
    g.close()


@pytest.mark.parametrize("group_size", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("lanes", [(16, 16), (32, 32)])
def test_group_sizes_and_lanes(group_size, lanes):
    """Chains cut in groups of 1 to 8 atoms in water, with exclusion masks: the
    pair kernel's builds with energies and stress (those without: below)."""
    from orac_b200.engine import Engine

    s = systems.solvated_chains(2100, 31, group_size=group_size)
    o, g = oracle.Oracle(s.copy()), Engine(s.copy())
    g.set_pair_tuning(*lanes, 5)
    o.update_lists()
    g.update_lists()
    for sh in "mlh":
        Fr, uer, sr = o.shell(sh)
        Fg, en, sg = g.shell(sh)
        assert rel_rms(Fg, Fr) <= 1e-5
        assert np.abs(g.ue6(en) - uer).max() <= 1e-6 * np.abs(uer).sum()
        assert np.linalg.norm(sg - sr) <= 1e-5 * np.linalg.norm(sr)
    g.close()


@pytest.mark.parametrize("variant", ["std", "rem", "alchemy"])
def test_forces_do_not_depend_on_energies_or_lanes(variant):
    """The same forces bit for bit with and without energies and for every
    launch configuration."""
    import torch

    from orac_b200.engine import Engine

    s = systems.ligand_in_water(nlig=13, nwat=1000, box=31.3, nfft=(32, 32, 32))
    s.ncell = (systems.linked_cells_for(31.3, s.shells),) * 3
    got = {}
    for cfg in ((16, 16, 5), (32, 32, 5), (16, 32, 6), (32, 16, 8)):
        g = Engine(s.copy())
        if variant == "rem":
            g.set_rem((s.ss_alchemy == -2).astype(int), 0, 0.7)
        elif variant == "alchemy":
            g.set_alchemy(s.ss_alchemy, 0.5, 0.5)
            g.set_lambda(0.0, 0.3, 0.0, 0.6)
        g.set_pair_tuning(*cfg)
        g.update_lists()
        dev = torch.device("cuda", 0)
        x, gr, mo = (torch.from_numpy(np.concatenate(a)).to(dev) for a in (
            (g.xp0, g.yp0, g.zp0), (g.xpg, g.ypg, g.zpg), (g.xpcm, g.ypcm, g.zpcm)))
        for energies in (True, False):
            for sh in (b"m", b"l", b"h"):
                f = torch.zeros(3 * s.ntap, dtype=torch.float64, device=dev)
                e = torch.zeros(8, dtype=torch.float64, device=dev)
                torch.cuda.synchronize()
                rc = g.lib.orac_gpu_mts_forces_dev(g.ctx, sh, x.data_ptr(), gr.data_ptr(), mo.data_ptr(),
                                                   f.data_ptr(), e.data_ptr() if energies else None, None)
                assert rc == 0
                torch.cuda.synchronize()
                got.setdefault(sh, []).append(f.cpu().numpy())
        g.close()
    for sh, fs in got.items():
        assert np.abs(fs[0]).max() > 0
        for f in fs[1:]:
            assert np.array_equal(f, fs[0]), sh


@pytest.mark.parametrize("nfft,order", [((8, 9, 10), 4), ((27, 35, 20), 5), ((30, 7, 25), 6), ((48, 49, 48), 4),
                                        ((96, 96, 14), 8), ((160, 162, 9), 4), ((210, 8, 12), 7)])
def test_plane_fft_grids(nfft, order):
    """Odd axes, an odd number of x lines, planes at and beyond the shared
    memory that the plane kernel uses."""
    from orac_b200.engine import Engine

    rng = np.random.default_rng(sum(nfft))
    n = 300
    box = np.array([14.0, 15.0, 13.0])
    x = rng.uniform(-0.6, 0.6, (3, n)) * box[:, None]
    q = rng.normal(0, 0.4, n)
    q -= q.mean()
    s = systems.two_waters()
    g, o = Engine(s.copy()), oracle.Oracle(s.copy())
    a = (x[0], x[1], x[2], q, np.diag(1.0 / box), float(box.prod()), 0.5)
    Fg, eg, vg = g.do_pmesh_kspace(*a, order, nfft)
    Fr, er, vr = o.do_pmesh_kspace(*a, order, nfft)[:3]
    assert rel_rms(Fg, Fr) <= 1e-5
    assert abs(eg - er) <= 1e-6 * abs(er)
    assert np.linalg.norm(vg - np.asarray(vr).reshape(3, 3)) <= 1e-5 * np.linalg.norm(vr)
    g.close()


def test_plan_of_a_call_with_its_own_grid():
    """Calls with their own grids leave the context's grid and results as they
    are, and keep one plan's memory."""
    from orac_b200.engine import Engine

    s = systems.water_box(nwat=216, box=18.8, lattice=6, nfft=(20, 20, 20))
    s.ncell = None
    s.shells = small_shells()
    g = Engine(s.copy())
    F0, e0, _ = g.fft_pme()
    r = s.cartesian()
    a = (r[0], r[1], r[2], s.charge, 0.5 * s.oc.T, s.volume, s.alphal)
    own = g.do_pmesh_kspace(*a, s.order, s.nfft)
    A = g.do_pmesh_kspace(*a, 4, (24, 25, 27))
    size = g.footprint()
    B = g.do_pmesh_kspace(*a, 6, (20, 21, 18))
    A2 = g.do_pmesh_kspace(*a, 4, (24, 25, 27))
    assert g.footprint() == size
    assert np.array_equal(A[0], A2[0]) and not np.array_equal(A[0], B[0])
    assert rel_rms(own[0], F0) <= 1e-12 and abs(own[1] - e0) <= 1e-12 * abs(e0)
    F1, e1, _ = g.fft_pme()
    assert np.array_equal(F0, F1)
    with pytest.raises(Exception):
        g.do_pmesh_kspace(*a, 4, (22, 20, 20))  # 11 is no factor
    F2, _, _ = g.fft_pme()
    assert np.array_equal(F0, F2)
    g.close()


def _same_as_fresh(g, s, setup):
    """Context g, given topology s after others, against a fresh context, bit for bit."""
    from orac_b200.engine import Engine

    f = Engine(s.copy())
    setup(f)
    f.update_lists()
    g.update_lists()
    for sh in "mlh":
        Ff, ef, sf = f.shell(sh)
        Fg, eg, sg = g.shell(sh)
        assert np.abs(Ff).max() > 0 and np.array_equal(Fg, Ff), sh
        # (energies and stress: FP64 sums of atomics, in any order)
        assert np.allclose(g.ue6(eg), f.ue6(ef), rtol=1e-12, atol=1e-9)
        assert np.linalg.norm(sg - sf) <= 1e-10 * np.linalg.norm(sf)
    # (fixed-point charge grid, one thread's sums after it)
    assert np.array_equal(g.fft_pme()[0], f.fft_pme()[0])
    if s.has_intra():
        assert rel_rms(g.intra_n1()[0], f.intra_n1()[0]) <= 1e-12
    f.close()


def test_topologies_one_after_another():
    """One context that takes a small topology, a larger one, the larger one
    with alchemy, a smaller one and its own again: what the earlier ones left
    (group records, selections by atom, bonded terms, MD state) neither stays
    in use nor sizes what follows."""
    from orac_b200.engine import Engine
    from orac_b200.lib import OracGpuError

    def take(g, s):
        g.s = s.copy()
        g._upload()

    def alch(e):
        e.set_alchemy(e.s.ss_alchemy, 0.5, 0.5)
        e.set_lambda(0.0, 0.3, 0.0, 0.6)

    def rem(e):
        e.set_rem(np.arange(e.s.ntap) % 5 == 0, 0, 0.7)

    def none(e):
        pass

    small = systems.water_box(nwat=64, box=18.8, lattice=5, nfft=(20, 20, 20))
    small.ncell = None
    small.shells = small_shells()
    chains = systems.solvated_chains(2100, 31)
    ligand = systems.ligand_in_water(nlig=13, nwat=1000, box=31.3, nfft=(32, 32, 32))
    ligand.ncell = (systems.linked_cells_for(31.3, ligand.shells),) * 3
    g = Engine(small.copy())
    rem(g)
    _same_as_fresh(g, small, rem)
    take(g, chains)  # larger: the selection by atom is gone
    _same_as_fresh(g, chains, none)
    g.md_setup(4.0, 2, 4, 6, "l")
    g.md_run(1)
    take(g, ligand)
    with pytest.raises(OracGpuError, match="md_setup"):
        g.md_run(1)
    _same_as_fresh(g, ligand, none)
    alch(g)
    _same_as_fresh(g, ligand, alch)
    take(g, ligand)  # the same number of atoms: the selection stays
    _same_as_fresh(g, ligand, alch)
    other = ligand.copy()  # other charges and a fixed mass
    other.charge = 0.9 * other.charge
    other.mass[5] = 1e25
    take(g, other)
    _same_as_fresh(g, other, alch)
    take(g, ligand)
    g.md_setup(4.0, 2, 4, 6, "l")
    g.md_run(1)
    take(g, small)
    _same_as_fresh(g, small, none)
    take(g, chains)
    _same_as_fresh(g, chains, none)
    g.close()


def _shell_dev(g, sh, energies=False):
    """Forces (3, N) of one shell through orac_gpu_mts_forces_dev."""
    import torch

    dev = torch.device("cuda", 0)
    x, gr, mo = (torch.from_numpy(np.concatenate(a)).to(dev) for a in (
        (g.xp0, g.yp0, g.zp0), (g.xpg, g.ypg, g.zpg), (g.xpcm, g.ypcm, g.zpcm)))
    f = torch.zeros(3 * g.s.ntap, dtype=torch.float64, device=dev)
    e = torch.zeros(8, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()
    rc = g.lib.orac_gpu_mts_forces_dev(g.ctx, sh.encode(), x.data_ptr(), gr.data_ptr(), mo.data_ptr(), f.data_ptr(),
                                       e.data_ptr() if energies else None, None)
    assert rc == 0
    torch.cuda.synchronize()
    return f.cpu().numpy().reshape(3, -1)


def _exclusions(s):
    out, p = [[] for _ in range(s.ntap)], 0
    for i in range(s.ntap):
        for j in s.mapnl[p + 1:p + 1 + s.mapnl[p]]:
            out[i].append(j - 1)
            out[j - 1].append(i)
        p += 1 + s.mapnl[p]
    return out


@pytest.mark.parametrize("group_size", [3, 4, 8])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("variant", ["std", "rem", "alchemy"])
def test_a_coordinate_that_is_no_number(group_size, value, variant):
    """An atom without coordinates spoils the forces of the groups in reach of
    its own (an evaluated pair with it, or the S'V share), and nothing else:
    not the atoms that follow a shorter group in the force array, not the
    atoms whose only pair with it is excluded."""
    from orac_b200.engine import Engine

    s = systems.solvated_chains(2100, 31, group_size=group_size)
    g = Engine(s.copy())
    if variant == "rem":
        g.set_rem(np.arange(s.ntap) % 5 == 0, 0, 0.7)
    elif variant == "alchemy":
        g.set_alchemy(np.where(np.arange(s.ntap) < 4, -2, 1), 0.5, 0.5)
        g.set_lambda(0.0, 0.3, 0.0, 0.6)
    g.update_lists()
    sh = s.shells
    first, last = s.grppt[:, 0] - 1, s.grppt[:, 1] - 1
    excl = _exclusions(s)
    size = last - first + 1
    # atoms near the end of their group in a chain, and the last molecule's last
    for a in (22, 23, s.ntap - 1):
        grp = int(s.atomg[a]) - 1
        d = np.stack([g.xpg - g.xpg[grp], g.ypg - g.ypg[grp], g.zpg - g.zpg[grp]])
        r = np.linalg.norm(np.asarray(s.co) @ (d - 2.0 * np.round(0.5 * d)), axis=0)
        far, masked = {}, []
        for k, ro, to, ri in (("m", sh.rcutm, sh.rtolm, 0.0), ("l", sh.rcutl, sh.rtoll, sh.rcutm)):
            near = (r < ro + to) & (r >= ri)
            near[grp] = True
            far[k] = ~np.repeat(near, size)
        for b in excl[a]:  # in the unswitched band of the M shell
            j = int(s.atomg[b]) - 1
            if j != grp and r[j] < sh.rcutm:
                masked.append(b)
        clean = {k: [_shell_dev(g, k, e) for e in (False, True)] for k in "ml"}
        keep = g.xp0
        g.xp0 = keep.copy()
        g.xp0[a] = value
        for k in "ml":
            for e in (False, True):
                F = _shell_dev(g, k, e)
                c = clean[k][e]
                assert np.array_equal(F[:, far[k]], c[:, far[k]]), (k, a)
                if k == "m":
                    # an entry evaluated pair by pair rounds differently: a few
                    # FP32 roundings of forces no larger than the largest
                    assert np.abs(F - c)[:, masked].max(initial=0.0) <= 1e-6 * np.abs(c).max(), (k, a)
        g.xp0 = keep
        assert all(v.sum() > s.ntap // 2 for v in far.values())
        assert masked or group_size == 8 or a == s.ntap - 1
    g.close()


def test_reciprocal_forces_keep_their_precision():
    """Two real x lines share one transform, which costs some of its rounding:
    the forces are no further from 64 bits than with a line of its own in each
    (5.21e-7, mean over 8 sets of charges of the same kind, standard error 1e-8),
    the cheaper transform's loss of 3% made up for in the gather."""
    from orac_b200 import units
    from orac_b200.engine import Engine

    s = systems.two_waters()
    g, o = Engine(s.copy()), oracle.Oracle(s.copy())
    err = []
    for seed in range(8):
        rng = np.random.default_rng([seed, 5])
        n = 9000
        edge = (n / 0.1) ** (1.0 / 3.0)
        x = rng.uniform(-0.5, 0.5, (3, n)) * edge
        q = rng.normal(0.0, 0.4, n)
        q = (q - q.mean()) * units.charge_internal(1.0)
        a = (x[0], x[1], x[2], q, np.eye(3) / edge, edge ** 3, 0.35, 4, (48, 48, 48))
        err.append(rel_rms(g.do_pmesh_kspace(*a)[0], o.do_pmesh_kspace(*a)[0]))
    assert np.mean(err) <= 5.21e-7, err
    g.close()


FORMS = {"soft": {}, "shift": dict(shifted=True, qshift=4.0, ljshift=0.35)}


def _chains(group_size, box="cubic"):
    """Chains in water; skewed: a sheared box, and some atoms of fixed mass."""
    s = systems.solvated_chains(2100, 31, group_size=group_size)
    s.ss_alchemy = np.where(np.arange(s.ntap) < 14, -2, np.where(np.arange(s.ntap) < 20, 2, 1)).astype(np.int32)
    s.rematom = (np.arange(s.ntap) % 5 == 0).astype(np.uint8)
    if box == "skewed":
        s.co = s.co.copy()
        s.co[0, 1], s.co[0, 2], s.co[1, 2] = 0.12 * s.co[0, 0], -0.08 * s.co[0, 0], 0.1 * s.co[0, 0]
        s.mass = s.mass.copy()
        s.mass[8:30] = 1e25
        s.ncell = None
    return s


def _variant(e, variant):
    if variant == "rem":
        e.set_rem(e.s.rematom, 0, 0.7)
    elif variant in FORMS:
        e.set_alchemy(e.s.ss_alchemy, 0.5, 0.5, **FORMS[variant])
        e.set_lambda(ladd=0.3, lrm=0.6, laddq=0.4, lrmq=0.7)


@pytest.mark.parametrize("box", ["cubic", "skewed"])
@pytest.mark.parametrize("variant", ["std", "rem", "soft", "shift"])
@pytest.mark.parametrize("group_size", [3, 4, 5, 8])
def test_builds_agree_bit_for_bit(group_size, variant, box):
    """Every build of the pair kernel for a group size and a variant -- with
    energies and without, half and whole warps, each number of blocks per SM --
    gives the same forces, and those of the oracle; in a skewed box, and with
    fixed masses, whose pairs alchemy skips."""
    from orac_b200.engine import Engine

    s = _chains(group_size, box)
    o = oracle.Oracle(s.copy())
    _variant(o, variant)
    o.update_lists()
    first = {}
    cfgs = ((16, 16, 5), (32, 32, 5), (16, 32, 6), (32, 16, 8)) if group_size <= 4 else ((32, 32, 5),)
    for cfg in cfgs:
        g = Engine(s.copy())
        _variant(g, variant)
        g.set_pair_tuning(*cfg)
        g.update_lists()
        for energies in (False, True):
            for sh in "mlh":
                F = _shell_dev(g, sh, energies)
                first.setdefault(sh, F)
                assert np.array_equal(F, first[sh]), (sh, cfg, energies)
        g.close()
    for sh in "mlh":
        assert rel_rms(first[sh], o.shell(sh)[0]) <= 1e-5, sh


@pytest.mark.parametrize("form", sorted(FORMS))
def test_energy_steps_do_not_change_a_schedules_trajectory(form):
    """The build that sums the work of a schedule (plain steps) and the one
    with energies (energy steps) give the same forces bit for bit."""
    from orac_b200.engine import Engine

    s = systems.ligand_in_water(nlig=13, nwat=1000, box=31.3, nfft=(32, 32, 32))
    s.ncell = (systems.linked_cells_for(31.3, s.shells),) * 3
    out = []
    for every in (0, 1, 3):
        g = Engine(s.copy())
        g.set_alchemy(s.ss_alchemy, 0.5, 0.5, **FORMS[form])
        g.set_lambda(0.0, 0.0, 0.0, 0.0)
        g.set_schedule([0.0, 40.0, 80.0], [1.0] * 3, [1.0] * 3, [0.0, 0.0, 1.0], [0.0, 1.0, 1.0])
        g.md_setup(4.0, 2, 4, 3, "l")
        g.md_run(14, energy_every=every)
        out.append(np.concatenate(g.md_state()))
        g.close()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("cells", [True, False])
def test_rows_longer_than_the_buffer(cells):
    """Rows of up to 700 partners, by linked cells and from all pairs: beyond
    the 512 that a warp gathers in shared memory."""
    from orac_b200.engine import Engine

    s = systems.water_box(nwat=1728, box=35.76, lattice=12, nfft=(40, 40, 40))
    s.shells = systems.Shells(rcutm=4.5, rtolm=0.3, rneim=0.4, rcutl=7.0, rtoll=0.3, rneil=0.5, rcuth=16.0, rtolh=0.3,
                              rneih=0.8)
    s.ncell = (systems.linked_cells_for(35.76, s.shells),) * 3 if cells else None
    o, g = oracle.Oracle(s.copy()), Engine(s.copy())
    o.update_lists()
    g.update_lists()
    # rows of the lower index: the first groups' hold all their neighbours
    c = np.stack(s.group_centres())
    d = c[:, :8, None] - c[:, None, :]
    d = np.einsum("ij,jab->iab", s.co, d - 2.0 * np.round(0.5 * d))
    assert ((d ** 2).sum(0) < 17.1 ** 2).sum(1).max() - 8 > 512
    pairs, _ = g.list_pairs()
    for sh in "hlm":
        assert pairs[sh] == len(o.lists[sh]) - s.ngrp, sh
    for sh in "mlh":
        F, Fr = _shell_dev(g, sh), o.shell(sh)[0]
        assert rel_rms(F, Fr) <= 1e-5, sh
    g.close()


def test_list_that_outgrows_its_capacity_in_a_run():
    """A state much denser than the one the lists were sized for: the rows that
    find no room are left out and the run reports it, also from a step graph."""
    from orac_b200.engine import Engine
    from orac_b200.lib import OracGpuError

    s = systems.water_box(nwat=1728, box=72.0, lattice=12, nfft=(48, 48, 48))
    s.shells = systems.Shells(rcutm=4.0, rtolm=0.3, rneim=0.4, rcutl=6.0, rtoll=0.3, rneil=0.4, rcuth=8.0, rtolh=0.3,
                              rneih=0.6)
    s.ncell = (systems.linked_cells_for(72.0, s.shells),) * 3
    g = Engine(s)
    g.md_setup(1.0, 2, 2, 2, "l")
    g.md_run(2)
    x, v = g.md_state()
    com = np.stack([np.bincount(s.atomp - 1, weights=s.mass * x[k]) / np.bincount(s.atomp - 1, weights=s.mass)
                    for k in range(3)])
    y = x + (0.65 - 1.0) * com[:, s.atomp - 1]  # (molecules as a whole, towards the box's centre)
    assert g.lib.orac_gpu_md_set_state(g.ctx, *[a.ctypes.data for a in (*np.ascontiguousarray(y),
                                                                       *np.ascontiguousarray(v))]) == 0
    with pytest.raises(OracGpuError, match="neighbour list capacity"):
        g.md_run(3)  # (lists are updated every second step, from the step before's centres)
    # set up again for the state at hand, the run goes on
    s.xyz_restart = np.ascontiguousarray(y)
    g.md_setup(1.0, 2, 2, 2, "l")
    g.md_run(3)
    assert np.isfinite(g.md_state()[0]).all()
    g.close()
