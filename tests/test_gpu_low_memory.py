"""Calls that go on with less when device memory runs short, outside an arena: the failed allocation
must not surface in a later launch check. The device is filled (with idle arenas) up to 8 MB: the
totals of 400 atoms and 450,000 k vectors fit their tables there (1.6 MB) but not the partial
structure factors of two chunks (14.5 MB, of a replica's one 7.2 MB), so they write S(k) in place. With
nothing free a box keeps the tile path.

The sums are added up in the same order whatever the room: equal to the last bit."""
import contextlib

import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _full_device(grx_lib, leave):
    """All but about `leave` bytes of device memory held."""
    free = grx_lib.Arena(leave) if leave else None
    held, size = [], 1 << 38
    while size >= 1 << 20:
        try:
            held.append(grx_lib.Arena(size))
        except RuntimeError:
            size >>= 1
    if free:
        free.close()
    try:
        yield
    finally:
        for a in held:
            a.close()


def _system(cells, kmax, nfw=400):
    s = synth.silica_co2(cells=cells, kmax=kmax)
    s["molsize"] = [400, 3]
    synth._set_atoms(s, s["pos"][:nfw], s["type"][:nfw], s["charge"][:nfw], [np.zeros((0, 3))])
    if nfw:
        synth.place_molecules(s, 1, 2, np.random.Generator(np.random.Philox(3)))
    return s


@pytest.mark.parametrize("replica", [0, 1])
def test_totals_go_on_in_place(grx_lib, replica):
    s = _system((1, 1, 2), (60, 60, 60))
    ref = grx_lib.Box(s, capacity=[400, 64])
    want, s_want = ref.total_energy(), ref.structure_factors()
    assert ref.ewald_sizes()[1] > 400000
    box = ref.replica() if replica else grx_lib.Box(s, capacity=[400, 64])
    with _full_device(grx_lib, (4 if replica else 8) << 20):
        got = box.total_energy()
    assert got == want
    for x, y in zip(box.structure_factors(), s_want):
        assert np.array_equal(x, y)


def test_box_without_room_to_build_lists(grx_lib):
    s = _system((4, 4, 6), (2, 2, 2))
    ref = grx_lib.Box(s, capacity=[400, 64])
    dims = ref.voxel_lists()[1]
    assert 16 * dims[0] * dims[1] * dims[2] > 2 << 20  # the counts of the voxels, in scratch
    ref.set_voxel_lists(0)
    rng = np.random.default_rng(4)
    pos = s["pos"][rng.integers(0, 400, 20)] + rng.uniform(-4, 4, (20, 3))
    args = (pos, np.full(20, -0.35), np.full(20, 3), 10 ** 6, 20, 1, 1)
    want, flags = ref.trial_energies(*args)
    box = grx_lib.Box(_system((4, 4, 6), (2, 2, 2), 0), capacity=[400, 64])
    box.set_voxel_lists(0)
    box.system = s
    box.set_component(0)
    box.set_component(1)
    with _full_device(grx_lib, 0):
        box.set_voxel_lists(1)
        assert not box.voxel_lists()[0]
        got, f = box.trial_energies(*args)
    assert np.array_equal(f, flags)
    ok = flags == 0
    assert ok.sum() >= 5 and np.array_equal(got[ok], want[ok])
