"""GPU parity of interaction::Tabulated (VerletListTabulated, FixedPairListTabulated)
against the oracle, and the reference's tabulated step-0 energies
(testsuite/tabulated/result.dat)."""
import math

import numpy as np
import pytest

from espressopp_b200 import _abi, interaction
from simdriver import (Sim, cell_grid, cuda_lib, lattice, load_polymer40k, mb_velocities,
                       oracle_lib, polymer_tab_tables, read_tab, write_tab_file)

pytestmark = pytest.mark.gpu

RC_SOFT = 2.5


def _rel_rms(a, b):
    return math.sqrt(np.sum((a - b) ** 2) / np.sum(b ** 2))


def _tab_pair(s, t1, t2, itype, tab, rc, shift=0.0):
    r, e, f = tab
    _abi.call(s.lib, "espp_tab_pair_set", s.h, t1, t2, itype, len(r), _abi.dptr(r),
              _abi.dptr(e), _abi.dptr(f), rc, shift)


def _tab_bond(s, itype, tab, rc=math.inf):
    r, e, f = tab
    _abi.call(s.lib, "espp_tab_bond_set", s.h, itype, len(r), _abi.dptr(r), _abi.dptr(e),
              _abi.dptr(f), rc, 0.0)


def _polymer(lib, prec, tabs, itype=2):
    pos, bonds, box, gold = load_polymer40k()
    s = Sim(lib, box, 0.3, cell_grid(box, 1.12, 0.3), precision=prec, seed=5)
    s.add(np.arange(1, len(pos) + 1), pos)
    s.decompose()
    s.vl(1.42)
    s.bonds(bonds)
    _tab_pair(s, 0, 0, itype, tabs[0], 1.12)
    _tab_bond(s, itype, tabs[1])
    return s, gold


@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_MIXED])
def test_tabulated_polymer_melt_golden_step0(tmp_path, prec):
    tl, tf, _, _ = polymer_tab_tables(tmp_path, cuda_lib())
    s, gold = _polymer(cuda_lib(), prec, (tl, tf))
    g = gold["tabulated"]
    assert round(s.energy(_abi.IA_TAB_PAIR), 3) == g["epair"]
    assert round(s.energy(_abi.IA_TAB_BOND), 3) == g["ebond"]


@pytest.mark.parametrize("itype", [1, 2, 3])
def test_tabulated_forces_and_observables_match_oracle(tmp_path, itype):
    tl, tf, _, _ = polymer_tab_tables(tmp_path, oracle_lib())
    o, _ = _polymer(oracle_lib(), _abi.PREC_FP64, (tl, tf), itype)
    g64, _ = _polymer(cuda_lib(), _abi.PREC_FP64, (tl, tf), itype)
    gmx, _ = _polymer(cuda_lib(), _abi.PREC_MIXED, (tl, tf), itype)
    ids = np.arange(1, 40001)
    for s in (o, g64, gmx):
        s.integrator(0.01)
        s.run(0)
    fo = o.particles(ids)[2]
    assert _rel_rms(g64.particles(ids)[2], fo) < 1e-12
    assert _rel_rms(gmx.particles(ids)[2], fo) < 1e-9
    # the bond list's long-time maximum, raised by the tabulated bond pass on FP64
    # distances in both precisions
    mx = np.zeros(3)
    for k, s in enumerate((o, g64, gmx)):
        _abi.call(s.lib, "espp_bonds_max_sqr", s.h, _abi.dptr(mx[k:]))
    assert mx[0] > 0 and np.all(np.abs(mx[1:] - mx[0]) <= 1e-14 * mx[0])
    for which in (_abi.IA_TAB_PAIR, _abi.IA_TAB_BOND):
        eo, wo = o.energy(which), o.virial(which)
        for g in (g64, gmx):
            assert abs(g.energy(which) - eo) < 1e-10 * abs(eo)
            assert abs(g.virial(which) - wo) < 1e-10 * abs(wo)
        assert np.allclose(g64.virial_tensor(which), o.virial_tensor(which), rtol=1e-9,
                           atol=1e-9)


def test_tabulated_langevin_run_matches_oracle(tmp_path):
    tl, tf, _, _ = polymer_tab_tables(tmp_path, oracle_lib())
    sims = [_polymer(oracle_lib(), _abi.PREC_FP64, (tl, tf), 3)[0],
            _polymer(cuda_lib(), _abi.PREC_FP64, (tl, tf), 3)[0],
            _polymer(cuda_lib(), _abi.PREC_MIXED, (tl, tf), 3)[0]]
    ids = np.arange(1, 40001)
    for s in sims:
        s.integrator(0.002)
        s.langevin(1.0, 1.0)
        s.run(30)
    ref = sims[0].particles(ids)
    for s, tol in ((sims[1], 1e-9), (sims[2], 1e-5)):
        got = s.particles(ids)
        assert np.max(np.abs(got[0] - ref[0])) < tol
        assert _rel_rms(got[1], ref[1]) < tol
    assert sims[1].num_resorts() == sims[0].num_resorts()


def test_lj_and_tabulated_on_one_verlet_list(tmp_path):
    """Two types: (0,0) Lennard-Jones, (0,1) and (1,1) tabulated; energies per interaction
    and the forces of both interactions together match the oracle."""
    pos, box = lattice(14, 0.8442, 0.05, seed=3)
    n = len(pos)
    types = (np.arange(n) % 3 == 0).astype(np.int32)
    vel = mb_velocities(n, 1.0, seed=4)
    soft = interaction.LennardJones(0.7, 1.1, cutoff=2.5)
    path = str(tmp_path / "soft.tab")
    write_tab_file(soft, path, N=400, low=0.6, high=2.6)
    tab = read_tab(oracle_lib(), path)
    sims = []
    for lib, prec in ((oracle_lib(), _abi.PREC_FP64), (cuda_lib(), _abi.PREC_FP64),
                      (cuda_lib(), _abi.PREC_MIXED)):
        s = Sim(lib, box, 0.3, cell_grid(box, 2.5, 0.3), precision=prec, seed=9)
        s.add(np.arange(n), pos, vel, types=types)
        s.decompose()
        s.vl(2.5)
        s.lj(0, 0, 1.0, 1.0, 2.5, 0.0)
        _tab_pair(s, 0, 1, 3, tab, 2.5, shift=0.01)
        _tab_pair(s, 1, 1, 1, tab, 2.2)
        s.integrator(0.004)
        s.run(0)
        sims.append(s)
    fo = sims[0].particles(np.arange(n))[2]
    assert _rel_rms(sims[1].particles(np.arange(n))[2], fo) < 1e-12
    assert _rel_rms(sims[2].particles(np.arange(n))[2], fo) < 1e-5
    for which in (_abi.IA_LJ, _abi.IA_TAB_PAIR):
        eo = sims[0].energy(which)
        for s in sims[1:]:
            assert abs(s.energy(which) - eo) < 1e-10 * abs(eo)
    for s in sims:
        s.run(25)
    ref = sims[0].particles(np.arange(n))
    got = sims[1].particles(np.arange(n))
    assert np.max(np.abs(got[0] - ref[0])) < 1e-9


def _soft_table(rc, strength):
    r = np.linspace(0.05, rc, 400)
    x = 1.0 - r / rc
    return r, strength * x ** 3, 3.0 * strength * x ** 2 / rc


def _two_types(n, seed):
    """A jittered lattice of n^3 points; every third particle has type 1."""
    pos, box = lattice(n, 0.8442, 0.1, seed)
    return pos, box, (np.arange(len(pos)) % 3 == 0).astype(np.int32)


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("prec,tol", [(_abi.PREC_FP64, 1e-12), (_abi.PREC_MIXED, 1e-8)])
def test_partners_of_a_type_without_a_table(prec, tol, late):
    """Only 0-0 pairs have a table; particles of type 1 are there when it is set, or come
    later.  Mixed: each of the ~30 contributing sums rounds once to 2^-32."""
    pos, box, typ = _two_types(12, 7)
    ids = np.arange(len(pos))
    out = []
    for lib, p in ((oracle_lib(), _abi.PREC_FP64), (cuda_lib(), prec)):
        s = Sim(lib, box, 0.3, cell_grid(box, 2.0, 0.3), precision=p, seed=5)
        first = typ == 0 if late else typ >= 0
        s.add(ids[first], pos[first], types=typ[first])
        s.decompose()
        s.vl(2.0)
        _tab_pair(s, 0, 0, _abi.TAB_LINEAR, _soft_table(2.0, 5.0), 2.0)
        if late:
            s.add(ids[typ == 1], pos[typ == 1], types=typ[typ == 1])
        s.integrator(0.002)
        s.run(0)
        out.append((s.particles(ids)[2], s.energy(_abi.IA_TAB_PAIR)))
    (fo, eo), (fg, eg) = out
    assert _rel_rms(fg, fo) < tol
    assert np.all(fg[typ == 1] == 0.0)
    assert abs(eg - eo) < 1e-10 * abs(eo)


def test_types_that_migrate_into_a_domain():
    """Two slab domains, a 0-0 table; the particles of type 1 start in the middle of one domain
    and drift into the other, which was set up without that type."""
    from espressopp_b200.domain import SpatialDecomposition

    pos, box = lattice(16, 0.8442, 0.05, 3)
    cg = cell_grid(box, RC_SOFT, 0.3)
    h = box[2] / cg[2]
    typ = ((pos[:, 2] > 1.4 * h) & (pos[:, 2] < 1.9 * h)).astype(np.int32)
    vel = np.zeros_like(pos)
    vel[typ == 1, 2] = 4.0
    ids = np.arange(len(pos), dtype=np.int64)
    r, e, f = _soft_table(RC_SOFT, 0.5)
    one = Sim(oracle_lib(), box, 0.3, cg, precision=_abi.PREC_FP64, seed=4)
    one.add(ids, pos, vel, typ)
    one.decompose()
    one.vl(RC_SOFT)
    _tab_pair(one, 0, 0, _abi.TAB_LINEAR, (r, e, f), RC_SOFT)
    one.integrator(0.005)
    dd = SpatialDecomposition(box, 0.3, cg, 2, precision=_abi.PREC_FP64, seed=4, lib=cuda_lib())
    dd.add_particles(ids, pos, vel, typ)
    dd.decompose()
    dd.vl_create(RC_SOFT)
    dd.tab_pair_set(0, 0, _abi.TAB_LINEAR, r, e, f, RC_SOFT)
    dd.integrator_set(0.005)
    for s in (one, dd):
        s.run(120)
    assert np.max(one.particles(ids)[0][typ == 1, 2]) > 2.5 * h
    (xo, _, fo, _), (xd, _, fd, _) = one.particles(ids), dd.get_particles(ids)
    assert np.max(np.abs(fd - fo)) < 1e-9
    assert np.max(np.abs((xd - xo + box / 2) % box - box / 2)) < 1e-9


@pytest.mark.parametrize("itype", [1, 2, 3])
def test_force_of_dimers(itype):
    """A single pair's FP64 force is the reference's bit for bit (Tabulated.hpp:99-115,
    Interpolation*.hpp): every operation of dist * f(r) / r is rounded once."""
    box = np.full(3, 9.0)
    sims = []
    for lib in (cuda_lib(), oracle_lib()):
        s = Sim(lib, box, 0.3, [3, 3, 3], precision=_abi.PREC_FP64, seed=3)
        s.add(np.arange(2), np.array([[1.0, 1.0, 1.0], [2.0, 1.0, 1.0]]))
        s.decompose()
        s.vl(2.0)
        _tab_pair(s, 0, 0, itype, _soft_table(2.0, 5.0), 2.0)
        s.integrator(0.002)
        sims.append(s)
    for d in np.linspace(0.3, 1.9, 150):
        q = np.array([[1.0, 1.0, 1.0], [1.0 + 0.48 * d, 1.0 + 0.6 * d, 1.0 + 0.64 * d]])
        f = []
        for s in sims:
            _abi.call(s.lib, "espp_set_particles", s.h, 2, _abi.i64ptr(np.arange(2)),
                      _abi.dptr(q), None)
            s.run(0)
            f.append(s.particles(np.arange(2))[2])
        assert np.array_equal(*f), d


@pytest.mark.parametrize("prec,tol", [(_abi.PREC_FP64, 1e-12), (_abi.PREC_MIXED, 1e-8)])
def test_tabulated_bonds_alone(prec, tol):
    """Bonds with a table and no pair potential: the tabulated pass writes every force itself,
    over whatever a pass before it left.  Mixed: a force rounds once to 2^-32."""
    pos, box = lattice(11, 0.8442, 0.1, 9)
    n = len(pos)
    k = np.arange(0, n - 1)
    bonds = np.stack([k, k + 1], 1)[(k + 1) % 11 != 0][::2]  # half of the particles have none
    r = np.linspace(0.01, 6.0, 500)
    out = []
    for lib, p in ((oracle_lib(), _abi.PREC_FP64), (cuda_lib(), prec)):
        s = Sim(lib, box, 0.3, cell_grid(box, 1.5, 0.3), precision=p, seed=5)
        s.add(np.arange(n), pos)
        s.decompose()
        s.vl(1.5)
        s.bonds(bonds)
        s.integrator(0.002)
        for strength in (300.0, 5.0):
            _tab_bond(s, _abi.TAB_LINEAR, (r, strength * (r - 1.0) ** 2, -2 * strength * (r - 1.0)))
            s.run(0)
        s.run(20)
        out.append(s.particles(np.arange(n)))
    (xo, vo, fo, _), (xg, vg, fg, _) = out
    assert _rel_rms(fg, fo) < 100 * tol and np.max(np.abs(xg - xo)) < 100 * tol
    free = np.setdiff1d(np.arange(n), bonds)
    assert len(free) and np.all(fg[free] == 0.0)
