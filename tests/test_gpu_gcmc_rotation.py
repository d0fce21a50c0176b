"""Translations and rotations of molecules of up to the 32 atoms that one warp moves (the rotation's
three angles are formed on three of its lanes), and the move choice at its probabilities' edges, against the FP64 oracle: identical attempts and decisions. Positions within
1e-9 A: a rotation rounds 10 A to 2e-15 (FP64) or 1e-13 (double-float sine and cosine, 1e-14), 80
moves add up to 1e-11. Mixed energies agree to 1e-6 kT, so one decision in 80 departs with a
chance below 1e-4 on a seeded chain."""
import numpy as np
import pytest

from graspa_gb300 import synth
from tests.test_gpu_gcmc import params, run_pair
from tests.systems import co2_system

pytestmark = pytest.mark.gpu


def helix_system(ms):
    """Two helical molecules of ms beads (1.3 A radius, 5 A long) in the slit pores of the silica."""
    s = co2_system()
    t = np.arange(ms)
    q = np.where(t % 2, -0.05, 0.05)
    q[-1] -= q.sum()
    nfw = s["comp_start"][1]
    s["templates"][1] = dict(pos=np.stack([1.3 * np.cos(0.9 * t), 1.3 * np.sin(0.9 * t), 5.0 * t / ms], axis=1),
                             charge=q, type=np.where(t % 3, 3, 2), names=["C_co2"] * ms)
    s["molsize"] = [nfw, ms]
    assert synth.place_molecules(s, 1, 2, np.random.default_rng(7), min_dist=2.4) == 2
    return s


@pytest.mark.parametrize("prec", ["GRX_FP64", "GRX_MIXED"])
@pytest.mark.parametrize("ms", [2, 3, 31, 32])
def test_rotation_of_long_molecules(grx_lib, ms, prec):
    s = helix_system(ms)
    d = params(grx_lib, p_translation=0.3, p_rotation=1.0, p_reinsertion=1.0, max_rotation=0.1, max_translation=0.3,
               norient=2)
    box, st, ost, after = run_pair(grx_lib, s, d, 80, getattr(grx_lib, prec))
    assert list(st.attempts) == list(ost.attempts) and list(st.accepted) == list(ost.accepted)
    assert st.attempts[1] > 0 and st.accepted[1] > 0
    nfw = s["comp_start"][1]
    assert np.max(np.abs(box.positions(1) - after["pos"][nfw:])) <= 1e-9


@pytest.mark.parametrize("prec", ["GRX_FP64", "GRX_MIXED"])
@pytest.mark.parametrize("ms,norient", [(2, 1), (2, 64), (11, 1), (12, 1), (12, 11), (32, 4)])
def test_orientations_across_warps(grx_lib, ms, norient, prec):
    """Orientation beads at the edges of a warp's ten and of the block's eighty: 1, 64, 10, 11, 121
    and 124 beads, grown and retraced by reinsertions."""
    s = helix_system(ms)
    d = params(grx_lib, p_translation=0.2, p_rotation=0.4, p_reinsertion=1.0, max_rotation=0.1, max_translation=0.3,
               norient=norient)
    box, st, ost, after = run_pair(grx_lib, s, d, 60, getattr(grx_lib, prec))
    assert list(st.attempts) == list(ost.attempts) and list(st.accepted) == list(ost.accepted)
    assert st.attempts[4] > 20
    assert np.max(np.abs(box.positions(1) - after["pos"][s["comp_start"][1]:])) <= 1e-9


@pytest.mark.parametrize("edges", [(0.0, 0.0, 0.0, 1.0), (0.0, 1.0, 1.0, 1.0), (0.1, 0.1, 0.1, 0.1), (1.0, 1.0, 1.0, 1.0),
                                   (-1.0, 0.3, 0.3, 7.0)])
def test_move_choice_edges(grx_lib, edges):
    s = co2_system(n_co2=3)
    d = params(grx_lib, p_translation=edges[0], p_rotation=edges[1], p_reinsertion=edges[2], p_swap=edges[3],
               pressure_pa=1e6)
    _, st, ost, _ = run_pair(grx_lib, s, d, 60, grx_lib.GRX_FP64)
    assert list(st.attempts) == list(ost.attempts) and list(st.accepted) == list(ost.accepted)
    assert st.n_molecules == ost.n_molecules
