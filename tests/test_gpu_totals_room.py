"""Totals in an arena with no room for the partial structure factors of the atom chunks: the sums are
added up in the same order as with room, so energies and structure factors are equal to the last bit
(a served job's arithmetic must not depend on what else is resident). Atom counts around the chunks
of 32 and more chunks than the eight sums they are spread over."""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfw,n_co2,kmax", [(3456, 3, (9, 9, 6)), (3456, 0, (9, 9, 6)), (577, 3, (9, 9, 14)), (1057, 11, (7, 5, 20))])
def test_sums_do_not_depend_on_room(grx_lib, nfw, n_co2, kmax):
    s = synth.silica_co2(kmax=kmax)
    s["molsize"] = [nfw, 3]
    synth._set_atoms(s, s["pos"][:nfw], s["type"][:nfw], s["charge"][:nfw], [np.zeros((0, 3))])
    if n_co2:
        synth.place_molecules(s, 1, n_co2, np.random.Generator(np.random.Philox(3)))
    cap = [nfw, 64]
    roomy = grx_lib.Arena(256 << 20)
    box = grx_lib.Box(s, capacity=cap, arena=roomy)
    box.set_voxel_lists(0)
    used = roomy.usage()[0]  # with the first scratch of 1 MB
    want, s_want = box.total_energy(), box.structure_factors()
    natoms = s["comp_start"][2]
    tables = 16 * (sum(kmax) + 3) * natoms + (160 << 10)  # of the atoms, and the results
    tight = grx_lib.Arena(used + max(0, tables - (1 << 20)) + (16 << 10))
    assert roomy.usage()[0] > tight.usage()[1]  # no room for the partial sums
    b = grx_lib.Box(s, capacity=cap, arena=tight)
    b.set_voxel_lists(0)
    assert b.total_energy() == want
    for x, y in zip(b.structure_factors(), s_want):
        assert np.array_equal(x, y)
    b.close()
    tight.close()
    box.close()
    roomy.close()
