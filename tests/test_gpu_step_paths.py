"""The step kernel's work splits at the sizes where they change: forces
against the FP64 oracle (bars of test_gpu_parity.py) and short trajectories
with the same bits whatever the launch shape."""
import numpy as np
import pytest

from md_nucleation_b200 import abi
from md_nucleation_b200 import generate as g
from tests.gpu_helpers import force_ok, forces_of, need_gpu, rel_rms

pytestmark = pytest.mark.gpu

CHECKED = abi.Q_ALL & ~abi.Q_BLIND_INSERT


@pytest.fixture(scope="module")
def eng():
    return need_gpu()


# core pairs: tiles of 32 atoms, ion and vapor in one tile or apart, a lone
# ion atom short of, on and past the edge
@pytest.mark.parametrize("n_vap", [0, 25])
@pytest.mark.parametrize("chain", [31, 32, 33, 64, 65])
@pytest.mark.parametrize("force_mode", [0, 1])
def test_core_tile_edges(eng, oracle_libs, chain, n_vap, force_mode):
    spec = g.small_system(seed=chain, gas="He", vapor="water", ion="chain", chain_atoms=chain, n_gas=300,
                          n_vap=n_vap, box=242.0)
    o = oracle_libs.OracleReplica(spec)
    o.step(3)
    e = eng.Engine([spec], force_mode=force_mode)
    e.upload(0, o.get_state())
    for term in (abi.I_AMBER, abi.I_VI, abi.I_VV, 0):
        e.compute_forces(term)
        Uo = o.compute_forces(term)
        a, b = forces_of(e.state(0), spec), forces_of(o.get_state(), spec)
        ok, err, rms = force_ok(a, b)
        assert ok, (term, err, rms)
        assert np.abs(e.energies()[0] - Uo).max() <= 1e-4 * max(np.abs(Uo).max(), 1e-6)
    if force_mode:
        assert rel_rms(a, b) <= 1e-9
