"""FP64 totals (structure factors by columns and atom chunks, tiled exclusions, guest atoms through
the trial pass) against the FP64 oracle at the edges of their tiles: framework sizes around 64-atom
exclusion tiles and 32-atom chunks, few and many k rows, framework pairs of several molecules,
replicas, and structure factors written in place when the arena has no room for partial sums.

Bars: |dS| <= 1e-10 (the reference's own check), and per total 1e-12 of the sum of the magnitudes
that cancel in it (pairs at prefactor |q_i q_j| / r; the largest Fourier total).
"""
import numpy as np
import pytest

from graspa_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

KEYS = ("hh_vdw", "hh_real", "hg_vdw", "hg_real", "gg_vdw", "gg_real")


def _system(nfw, n_co2, kmax=(4, 5, 6), molecules=1):
    """The first nfw framework atoms of a small silica cell (as `molecules` molecule ids) and CO2."""
    s = synth.silica_co2(cells=(1, 1, 2), kmax=kmax)
    fw = slice(0, nfw)
    s["molsize"] = [nfw // molecules, 3]
    synth._set_atoms(s, s["pos"][fw], s["type"][fw], s["charge"][fw], [np.zeros((0, 3))])
    if n_co2:
        synth.place_molecules(s, 1, n_co2, np.random.Generator(np.random.Philox(3)))
    s["molid"][:nfw] = np.arange(nfw) // s["molsize"][0]
    return s


def _check(grx_lib, box, s, exclusions=True):
    S = O.OracleSystem(s)
    ref, s_fw, s_ads = S.ewald_total(s["molsize"])
    t, ovl = box.total_energy(with_overlap=True)
    pair = S.vdw_real_total()
    # magnitudes of the Coulomb sums: every pair at prefactor |q_i q_j| / r
    cell = np.array(s["cell"]).reshape(3, 3)
    f = (s["pos"][None, :, :] - s["pos"][:, None, :]) @ np.linalg.inv(cell)
    r = np.linalg.norm((f - np.round(f)) @ cell, axis=2) + np.eye(len(f)) * 1.0
    q = np.abs(s["charge"])
    q2 = s["prefactor"] * float((q[:, None] * q[None, :] / r).sum())
    for k, p in zip(KEYS, pair):
        assert abs(t[k] - p) <= 1e-12 * (1.0 + abs(p) + (q2 if k.endswith("real") else 0.0)), k
    ew = box.ewald_total()
    for k in range(7 if exclusions else 5):
        assert abs(ew[k] - ref[k]) <= 1e-12 * (1.0 + abs(ref[k]) + (q2 if k > 2 else abs(ref[:3]).max())), k
    assert int(ew[7]) == int(ref[7])
    a, b, c = box.structure_factors()
    _, act = S.ewald_active()
    m = np.repeat(act.astype(bool), 2)
    for got, want in ((a, s_fw), (b, s_ads), (c, s_ads)):
        assert np.max(np.abs(got - want)[m], initial=0.0) <= 1e-10
        assert not np.any(got[~m])
    assert ovl == 0


@pytest.mark.parametrize("nfw,n_co2,kmax", [(64, 2, (4, 5, 6)), (65, 1, (4, 5, 6)), (129, 0, (1, 1, 1)), (127, 3, (0, 2, 1)),
                                            (576, 4, (9, 9, 14)), (33, 2, (2, 0, 20))])
def test_totals_at_tile_edges(grx_lib, nfw, n_co2, kmax):
    s = _system(nfw, n_co2, kmax)
    box = grx_lib.Box(s, capacity=[nfw, 64])
    _check(grx_lib, box, s)
    if n_co2:  # a replica reads its parent's framework sums
        box.ewald_total()
        _check(grx_lib, box.replica(), s)


@pytest.mark.parametrize("molecules", [2, 9])
def test_totals_of_framework_molecules(grx_lib, molecules):
    s = _system(288, 3, molecules=molecules)
    # the pair totals; exclusions take consecutive stored atoms as a molecule, and framework atoms
    # are stored in k-d order
    _check(grx_lib, grx_lib.Box(s, capacity=[288, 64]), s, exclusions=False)


def test_structure_factors_in_place_without_room(grx_lib):
    s = synth.silica_co2(n_co2=3)
    cap = [s["comp_start"][1], 64]
    box = grx_lib.Box(s, capacity=cap)
    want = box.total_energy()
    s_want = box.structure_factors()
    probe = grx_lib.Arena(64 << 20)
    b = grx_lib.Box(s, capacity=cap, arena=probe)
    b.set_voxel_lists(0)
    used = probe.usage()[0]
    b.close()
    probe.close()
    arena = grx_lib.Arena(used + (2 << 20))  # tables of the atoms fit, partial sums of 100 chunks do not
    b = grx_lib.Box(s, capacity=cap, arena=arena)
    got = b.total_energy()
    for k in want:
        assert abs(got[k] - want[k]) <= 1e-12 * max(abs(want[k]), abs(want["gg_ewald"]) * 1e-2, 1.0), k
    for x, y in zip(b.structure_factors(), s_want):
        assert np.max(np.abs(x - y)) <= 1e-10
    b.close()
    arena.close()
