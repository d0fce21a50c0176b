"""Single-molecule deltas of one side (do_new = 0 or do_old = 0): the side that is left out may hold
anything (types past the pair tables, positions that are no numbers) and is not evaluated; the two
sides add up to the full delta, to the last bit. For adsorbate and framework molecules, the tile path
and voxel lists, and one and three beads."""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("lists", [0, 1])
@pytest.mark.parametrize("component,beads", [(1, 3), (1, 1), (0, 3)])
def test_sides_of_a_delta(grx_lib, component, beads, lists, prec):
    s = synth.silica_co2(n_co2=4)
    nfw = s["comp_start"][1]
    box = grx_lib.Box(s, capacity=[nfw, 64])
    box.set_voxel_lists(lists)
    p = grx_lib.PRECISIONS[prec]
    # a guest, or framework atoms next to one (they meet guests only)
    first = nfw if component else int(np.argmin(np.linalg.norm(s["pos"][:nfw - 2] - s["pos"][nfw], axis=1)))
    old = dict(pos=s["pos"][first:first + beads], charge=s["charge"][first:first + beads],
               type=s["type"][first:first + beads], molid=int(s["molid"][first]))
    new = dict(old, pos=old["pos"] + [0.3, -0.2, 0.1])
    junk = dict(pos=np.full((beads, 3), np.nan), charge=np.full(beads, np.nan), type=np.full(beads, 10 ** 8), molid=77)
    both, flag = box.single_body(old, new, component, prec=p)
    only_new, f_new = box.single_body(junk, new, component, do_old=0, prec=p)
    only_old, f_old = box.single_body(old, junk, component, do_new=0, prec=p)
    assert np.array_equal(only_new + only_old, both)
    assert np.any(only_new != 0) and np.any(only_old != 0)
    assert f_new == flag and f_old == 0


def test_any_other_precision_is_fp32(grx_lib):
    """The entry point takes every value past the two wider forms as FP32."""
    s = synth.silica_co2(n_co2=4)
    nfw = s["comp_start"][1]
    box = grx_lib.Box(s, capacity=[nfw, 64])
    old = dict(pos=s["pos"][nfw:nfw + 3], charge=s["charge"][nfw:nfw + 3], type=s["type"][nfw:nfw + 3], molid=0)
    new = dict(old, pos=old["pos"] + 0.2)
    want, _ = box.single_body(old, new, 1, prec=grx_lib.GRX_FP32)
    for prec in (3, 4, -1):
        assert np.array_equal(box.single_body(old, new, 1, prec=prec)[0], want), prec
