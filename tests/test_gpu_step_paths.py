"""The step kernel's work splits at the sizes where they change: forces
against the FP64 oracle (bars of test_gpu_parity.py) and short trajectories
with the same bits whatever the launch shape."""
import numpy as np
import pytest

from md_nucleation_b200 import abi
from md_nucleation_b200 import generate as g
from md_nucleation_b200.system import QQRD2E
from tests.gpu_helpers import FORCE_ATOL, forces_of, need_gpu, rel_rms

pytestmark = pytest.mark.gpu

CHECKED = abi.Q_ALL & ~abi.Q_BLIND_INSERT


@pytest.fixture(scope="module")
def eng():
    return need_gpu()


# core pairs: tiles of 32 atoms, ion and vapor in one tile or apart, a lone
# ion atom short of, on and past the edge.  Which pairs a tile takes is the
# same code for both precisions; FP64 shows a wrong pair to 1e-9.
@pytest.mark.parametrize("n_vap", [0, 25])
@pytest.mark.parametrize("chain", [31, 32, 33, 64, 65])
def test_core_tile_edges(eng, oracle_libs, chain, n_vap):
    spec = g.small_system(seed=chain, gas="He", vapor="water", ion="chain", chain_atoms=chain, n_gas=300,
                          n_vap=n_vap, box=242.0)
    o = oracle_libs.OracleReplica(spec)
    o.step(3)
    e = eng.Engine([spec], force_mode=1)
    e.upload(0, o.get_state())
    for term in (abi.I_AMBER, abi.I_VI, abi.I_VV, 0):
        e.compute_forces(term)
        Uo = o.compute_forces(term)
        a, b = forces_of(e.state(0), spec), forces_of(o.get_state(), spec)
        assert rel_rms(a, b) <= 1e-9 or np.sqrt(np.mean((a - b) ** 2)) <= FORCE_ATOL, term
        assert np.abs(e.energies()[0] - Uo).max() <= 1e-4 * max(np.abs(Uo).max(), 1e-6)


def _pair_bound(spec, st, term):
    """What FP32 pair terms may be off by, per atom and component, on top of a
    sum of FP64 pairs: u = 2^-24.  A pair's factor is a product of some 20
    operations and a reciprocal root of 3 u that enters 14 times, summed over
    at most 32 steps: 100 u of its terms.  Coordinates relative to the ion
    centre are rounded to u of their size, which changes the force by the
    displacement times (15, 9, 4) of the repulsive, dispersion and Coulomb
    factor (their derivatives, and the factor itself)."""
    vin = st.region[1 + spec.n_gas:].astype(bool)
    ni, av, nv = spec.ion.n, spec.vapor.n, int(vin.sum())
    x = np.concatenate([st.ion_x.reshape(-1, 3), st.vap_ax[vin].reshape(-1, 3)])
    t = np.concatenate([spec.ion.type, np.tile(spec.vapor.type, nv)])
    q = np.concatenate([spec.ion.charge, np.tile(spec.vapor.charge, nv)])
    w = np.concatenate([np.ones(ni), st.vap_w[vin].reshape(-1)])
    mol = np.concatenate([np.full(ni, -1), np.repeat(np.arange(nv), av)])
    ion = mol < 0
    if term == abi.I_AMBER:
        on = ion[:, None] & ion[None]
        np.fill_diagonal(on, False)
        for rows, k in ((spec.ion.bonds, 1), (spec.ion.rigid, 1), (spec.ion.angles, 2), (spec.ion.dihedrals, 3)):
            on[rows[:, 0], rows[:, k]] = on[rows[:, k], rows[:, 0]] = False
    elif term == abi.I_VI:
        on = ion[:, None] != ion[None]
    else:
        on = ~ion[:, None] & ~ion[None] & (mol[:, None] != mol[None])
    r = np.linalg.norm(x[:, None] - x[None], axis=2)
    r[~on] = 1.0
    eps = np.sqrt(spec.atom_eps[t][:, None] * spec.atom_eps[t][None])
    sig = 0.5 * (spec.atom_sigma[t][:, None] + spec.atom_sigma[t][None])
    ww = np.where(on, w[:, None] * w[None], 0.0)
    a, b = 48 * eps * sig ** 12 * r ** -14 * ww, 24 * eps * sig ** 6 * r ** -8 * ww
    c = np.abs(QQRD2E * q[:, None] * q[None]) * r ** -3 * ww
    com = np.average(x[:ni], axis=0, weights=spec.atom_mass[t[:ni]])
    far = np.linalg.norm(x - com, axis=1)
    u = 2.0 ** -24
    return u * (100 * (a + b + c) * r + (15 * a + 9 * b + 4 * c) * (far[:, None] + far[None])).sum(axis=1)


# The FP32 tile has loads, masks and packed arithmetic of its own: the same
# edges term by term, in the kernels with and without gas-gas terms, and the
# steps without energies (four pairs at once) against those with (two)
@pytest.mark.parametrize("gg", [False, True])
@pytest.mark.parametrize("n_vap", [0, 25])
@pytest.mark.parametrize("chain", [31, 32, 33, 64, 65])
def test_core_tile_edges_fp32(eng, oracle_libs, chain, n_vap, gg):
    spec = g.small_system(seed=chain, gas="He", vapor="water", ion="chain", chain_atoms=chain, n_gas=300,
                          n_vap=n_vap, box=242.0, gas_min_dist=4.0 if gg else 0.0)
    if gg:
        spec.interactions |= abi.I_GG
    o = oracle_libs.OracleReplica(spec)
    o.step(3)
    start = o.get_state()
    e = eng.Engine([spec])
    e.upload(0, start)
    gas = int(start.region[1:1 + spec.n_gas].sum()) * spec.gas.n
    for term in (abi.I_AMBER, abi.I_VI, abi.I_VV):
        e.compute_forces(term)
        o.compute_forces(term)
        a, b = forces_of(e.state(0), spec), forces_of(o.get_state(), spec)
        bound = np.insert(_pair_bound(spec, start, term), [spec.ion.n] * gas, 0.0)
        # and the fixed-point terms' rounding, the bonded terms' FP64
        err = np.abs(a - b).max(axis=1)
        assert (err <= bound + 1e-9 + 1e-11 * np.abs(b).max()).all(), (term, np.max(err - bound))
    out = []
    for mode in (0, 2):
        e.upload(0, start)
        e.step(3, mode)
        out.append(e.state(0))
    for x, y in zip(vars(out[0]).values(), vars(out[1]).values()):
        assert np.array_equal(x, y)


def _run(eng, spec, shapes, steps=12, **kw):
    """steps per launch shape (cluster, threads), from the spec's start."""
    e = eng.Engine([spec], quirks=CHECKED, **kw)
    for c, t in shapes:
        e.set_launch(c, t)
        e.step(steps, 1)
    s = e.state(0)
    return np.concatenate([a.ravel() for a in (s.ion_x, s.ion_v, s.ion_f, s.gas_ax, s.gas_av, s.gas_af, s.vap_ax,
                                               s.vap_av, s.vap_af, s.mol_x, e.energies())])


# near molecules: records built for one cluster size and used at another,
# none / one / many heavy molecules (more than 16 partners) for a warp, one
# and two gas atoms, a last group of a few lanes
@pytest.mark.parametrize("gas,chain,n_gas", [("He", 0, 60), ("Ar", 20, 3000), ("N2", 90, 5000), ("N2", 200, 2500)])
@pytest.mark.parametrize("force_mode", [0, 1])
def test_near_records_do_not_depend_on_the_launch(eng, gas, chain, n_gas, force_mode):
    spec = g.small_system(seed=5 + chain, gas=gas, vapor="methanol", ion="chain" if chain else "nacl",
                          chain_atoms=chain, n_gas=n_gas, n_vap=12, box=245.0, shake_h=True)
    a = _run(eng, spec, [(1, 512)] * 4, force_mode=force_mode)
    b = _run(eng, spec, [(8, 512), (1, 64), (3, 96), (2, 256)], force_mode=force_mode)
    assert np.array_equal(a, b)


# CTAs of one warp: fewer threads than build_near has bins
@pytest.mark.parametrize("gas,chain,n_gas", [("He", 0, 800), ("Ar", 20, 3000), ("N2", 90, 2500)])
@pytest.mark.parametrize("force_mode", [0, 1])
@pytest.mark.parametrize("gg", [False, True])
def test_one_warp_per_block(eng, gas, chain, n_gas, force_mode, gg):
    spec = g.small_system(seed=6 + chain, gas=gas, vapor="methanol", ion="chain" if chain else "nacl",
                          chain_atoms=chain, n_gas=n_gas, n_vap=12, box=245.0, shake_h=True,
                          gas_min_dist=4.0 if gg else 0.0)
    if gg:
        spec.interactions |= abi.I_GG
    spec.margin = 2.0  # rebuilds among the steps
    a = _run(eng, spec, [(1, 512)] * 3, steps=40, force_mode=force_mode)
    for c in (1, 8):
        assert np.array_equal(a, _run(eng, spec, [(c, 32)] * 3, steps=40, force_mode=force_mode))


# energies of every step and the thermostats, whose kicks and factors each
# thread applies to its own components: one CTA, two that exchange their sums,
# more that take slices of them
@pytest.mark.parametrize("mode", [abi.NVT_SCALE, abi.NVT_NH])
def test_thermostats_and_energies_do_not_depend_on_the_launch(eng, mode):
    spec = g.small_system(seed=33, gas="N2", vapor="water", ion="chain", chain_atoms=40, n_gas=2500, n_vap=30,
                          box=245.0, shake_h=True)
    out = []
    for c, t in ((1, 512), (2, 512), (5, 128), (8, 256)):
        e = eng.Engine([spec], quirks=CHECKED)
        e.set_nvt(mode, 310.0)
        e.set_launch(c, t)
        for _ in range(3):
            e.step(9, 2)
        s = e.state(0)
        out.append(np.concatenate([a.ravel() for a in (s.ion_x, s.ion_v, s.ion_f, s.gas_ax, s.gas_av, s.vap_ax,
                                                       s.vap_av, e.energies())]))
    assert all(np.array_equal(out[0], o) for o in out[1:])


def all_rigid(spec):
    """Every bond of the vapor a constraint: five that share atoms, more than
    the kernels solve as a group."""
    v = spec.vapor
    v.rigid = np.concatenate([v.rigid, v.bonds]).astype(np.int32)
    v.bonds = np.zeros((0, 3), np.int32)
    return spec


def test_large_constraint_groups_are_swept(eng, oracle_libs):
    spec = all_rigid(g.small_system(seed=17, gas="He", vapor="methanol", ion="nacl", n_gas=800, n_vap=20, box=242.0,
                                    shake_h=True))
    o = oracle_libs.OracleReplica(spec)
    out = []
    for c, t in ((1, 512), (8, 128)):
        e = eng.Engine([spec])
        e.set_launch(c, t)
        e.step(10)
        out.append(e.state(0))
        assert not e.status().any()
    assert np.array_equal(out[0].vap_ax, out[1].vap_ax)
    o.step(10)
    inside = out[0].region[1 + spec.n_gas:].astype(bool)
    assert inside.sum() >= 3
    # the bar of the short trajectories in test_gpu_parity.py
    assert np.abs(out[0].vap_ax[inside] - o.get_state().vap_ax[inside]).max() <= 1e-6
