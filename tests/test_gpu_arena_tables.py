"""FP64 tables of boxes in an arena: taken from the arena and counted in the footprint (no other device
memory is touched when a box comes or goes), shared by boxes of equal parameters until the last of
them goes, and part of the box: what does not fit is refused with nothing left allocated."""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu

CAP = [576, 64]


def _system(alpha=0.265):
    return synth.silica_co2(cells=(1, 1, 2), kmax=(5, 5, 6), n_co2=3, alpha=alpha)


def _box(grx_lib, arena, alpha=0.265):
    b = grx_lib.Box(_system(alpha), capacity=CAP, arena=arena)
    b.set_voxel_lists(0)
    return b


def _energies(grx_lib, box):
    rng = np.random.default_rng(3)
    pos = rng.uniform(0, 1, (16, 3)) @ np.array(box.system["cell"]).reshape(3, 3)
    return box.trial_energies(pos, np.full(16, -0.35), np.full(16, 3), 10 ** 6, 16, 1, 1, prec=grx_lib.GRX_FP64)[0]


def test_tables_come_from_the_arena(grx_lib):
    torch = pytest.importorskip("torch")
    arena = grx_lib.Arena(256 << 20)
    first = _box(grx_lib, arena, 0.2)
    _energies(grx_lib, first)
    free = torch.cuda.mem_get_info()[0]
    boxes = [_box(grx_lib, arena, 0.2 + 0.004 * k) for k in range(1, 21)]
    assert torch.cuda.mem_get_info()[0] > free - (4 << 20)  # 20 tables of 0.4 MB are 8 MB
    for k, b in enumerate(boxes):
        plain = grx_lib.Box(b.system, capacity=CAP)
        plain.set_voxel_lists(0)
        assert np.array_equal(_energies(grx_lib, b), _energies(grx_lib, plain)), k
        plain.close()
    for b in boxes + [first]:
        b.close()
    assert arena.usage()[0] == 0
    arena.close()


def test_shared_until_the_last_box_goes(grx_lib):
    arena = grx_lib.Arena(64 << 20)
    a = _box(grx_lib, arena)
    one = arena.usage()[0]
    want = _energies(grx_lib, a)
    b = _box(grx_lib, arena)
    assert one > arena.usage()[0] - one  # the second box without tables of its own
    a.close()
    c = _box(grx_lib, arena, 0.3)  # takes the memory of the first
    assert np.array_equal(_energies(grx_lib, b), want)
    b.close()
    c.close()
    assert arena.usage()[0] == 0
    arena.close()


def test_footprint_holds_the_tables(grx_lib):
    fp = grx_lib.box_footprint(_system(), CAP)
    arena = grx_lib.Arena(fp)
    b = _box(grx_lib, arena)
    used = arena.usage()[0]
    plain = grx_lib.Box(_system(), capacity=CAP)
    plain.set_voxel_lists(0)
    assert np.array_equal(_energies(grx_lib, b), _energies(grx_lib, plain))
    b.close()
    arena.close()
    small = grx_lib.Arena(used - 200_000)  # room for all but the tables
    with pytest.raises(grx_lib.GrxError, match="memory"):
        _box(grx_lib, small)
    assert small.usage()[0] == 0
    small.close()


def test_narrow_boxes_fit_by_their_footprint(grx_lib):
    """An arena of 24 footprints takes 24 boxes of a cell narrower than twice the list radius: no lists
    (4 to 9 MB a box) on top of the footprint."""
    fp = grx_lib.box_footprint(_system(), CAP)
    arena = grx_lib.Arena(24 * fp)
    boxes = [grx_lib.Box(_system(), capacity=CAP, arena=arena) for _ in range(24)]
    assert not any(b.voxel_lists()[0] for b in boxes)
    for b in boxes:
        b.close()
    arena.close()
