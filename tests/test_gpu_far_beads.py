"""Beads many cells from the home cell (unwrapped positions) on voxel lists and on tiles: pairs next to
the cutoff must survive the FP32 screen at any distance. Beads sit 1e-4 to 2e-3 A inside the cutoff of a
framework atom's image, up to 60 cells out (2,400 A), on a thinned framework (12 atoms, LJ unshifted),
so that one lost pair is a large part of a trial's energy.

Bars, with M the sum of the magnitudes of a trial's pair terms (no atom nearer than 9 A, where a term
changes by at most 2.5 of itself per A): a displacement at 2,400 A carries 1e-12 A on either side, so
1e-11 M for FP64; 1e-6 kT (and 1e-6 M) for the mixed form; the FP32 form keeps a displacement to 1e-6 A
and its functions to 1e-5: 1e-4 M. The smallest term of every trial is at least twice its bar (checked).
"""
import numpy as np
import pytest
from scipy.special import erfc

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu

LATTICES = [(0, 0, 0), (0, 0, 5), (12, 0, 0), (0, 0, 25), (0, 0, 40), (20, -20, 10), (-30, 25, 30), (0, 0, 60)]


def _system(which, path):
    """Twelve framework atoms of the system's framework (spread, or in a cluster: a tile with one image),
    no LJ shift."""
    s = {"silica": synth.silica_co2, "triclinic": lambda: synth.adsorbate_system("CO2", 3, n_atoms=1500),
         "skewed": lambda: synth.adsorbate_system("CO2", 11, n_atoms=1500)}[which]()
    n, rng = s["comp_start"][1], np.random.default_rng(2)
    keep = np.sort(rng.choice(n, 12, replace=False))
    if path == "tiles":
        middle = 0.5 * np.array(s["cell"]).reshape(3, 3).sum(0)
        keep = np.sort(np.argsort(np.linalg.norm(s["pos"][:n] - middle, axis=1))[:12])
    s["molsize"] = [12] + list(s["molsize"][1:])
    synth._set_atoms(s, s["pos"][keep], s["type"][keep], s["charge"][keep], [np.zeros((0, 3))])
    s["shift"] = np.zeros_like(s["shift"])
    return s


def _terms(s, p, q, ty):
    """(LJ, Coulomb) of every (bead, atom) pair inside the cutoff, and the distances; p in the home cell."""
    cell, nt = np.array(s["cell"]).reshape(3, 3), s["ntypes"]
    f = (s["pos"][None] - p[:, None]) @ np.linalg.inv(cell)
    r = np.linalg.norm((f - np.round(f)) @ cell, axis=2)
    row = (s["type"][None, :], ty[:, None])
    eps, sig = (np.asarray(s[k]).reshape(nt, nt)[row] for k in ("epsilon", "sigma"))
    t = (sig / r) ** 6
    lj = np.where(r < s["cutoff_vdw"], 4 * eps * (t * t - t), 0.0)
    co = np.where(r < s["cutoff_coul"], s["prefactor"] * s["charge"][None] * q[:, None] * erfc(s["alpha"] * r) / r, 0.0)
    return lj, co, r


@pytest.mark.parametrize("prec", ["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("which", ["silica", "triclinic", "skewed"])
@pytest.mark.parametrize("path", ["lists", "tiles"])
def test_pairs_at_the_cutoff_far_from_home(grx_lib, path, which, prec):
    s = _system(which, path)
    box = grx_lib.Box(s, capacity=[12, 64])
    assert box.voxel_lists()[0]
    if path == "tiles":
        box.set_voxel_lists(0)
    cell = np.array(s["cell"]).reshape(3, 3)
    rng = np.random.default_rng(9)
    n = 600
    v = rng.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    p = s["pos"][rng.integers(0, 12, n)] + (s["cutoff_coul"] - rng.uniform(1e-4, 2e-3, n))[:, None] * v
    f = p @ np.linalg.inv(cell)
    p = (f - np.floor(f)) @ cell
    tm = s["templates"][1]
    q, ty = np.full(n, tm["charge"][-1]), np.full(n, tm["type"][-1])
    lj, co, r = _terms(s, p, q, ty)
    least = np.where(co != 0, np.abs(co), np.inf).min(1)
    keep = (r.min(1) > 9.0) & (least > 0.01)
    p, q, ty, lj, co, least = p[keep], q[keep], ty[keep], lj[keep], co[keep], least[keep]
    n = len(p)
    assert n >= 60
    want = np.stack([lj.sum(1), co.sum(1)], 1)
    mag = np.stack([np.abs(lj).sum(1), np.abs(co).sum(1)], 1)
    bar = {"fp64": 1e-11 * mag, "mixed": np.maximum(1e-6 * mag, 1e-6 / grx_lib.beta_from_temperature(300.0)),
           "fp32": 1e-4 * mag}[prec]
    assert np.all(least > 2 * bar[:, 1])
    for lattice in LATTICES:
        e, _ = box.trial_energies(p + np.array(lattice) @ cell, q, ty, 10 ** 6, n, 1, 1, prec=grx_lib.PRECISIONS[prec])
        assert np.all(np.abs(e[:, :2] - want) <= bar), (lattice, int((np.abs(e[:, :2] - want) > bar).any(1).sum()))


def test_pairs_at_the_cutoff_in_a_wide_cell(grx_lib):
    """FP64 on tiles in a cell of 80,000 A, whose coordinates the hi parts hold to 4e-3 A only. Bar:
    displacements carry 1.5e-11 A, a term changes by at most 2.5 of itself per A: 1e-10 M."""
    s = _system("silica", "tiles")
    s["pos"] = s["pos"] - s["pos"][0] + np.array([70011.3, 68123.7, 71987.1])
    s["cell"] = synth.orthorhombic_cell(80000.0, 80000.0, 80000.0)
    box = grx_lib.Box(s, capacity=[12, 64])
    assert not box.voxel_lists()[0]
    rng = np.random.default_rng(9)
    n = 400
    v = rng.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    p = s["pos"][rng.integers(0, 12, n)] + (s["cutoff_coul"] - rng.uniform(1e-4, 2e-3, n))[:, None] * v
    tm = s["templates"][1]
    q, ty = np.full(n, tm["charge"][-1]), np.full(n, tm["type"][-1])
    lj, co, r = _terms(s, p, q, ty)
    k = r.min(1) > 9.0
    assert k.sum() >= 60
    e, _ = box.trial_energies(p[k], q[k], ty[k], 10 ** 6, int(k.sum()), 1, 1, prec=grx_lib.GRX_FP64)
    want = np.stack([lj[k].sum(1), co[k].sum(1)], 1)
    mag = np.stack([np.abs(lj[k]).sum(1), np.abs(co[k]).sum(1)], 1)
    assert np.all(np.abs(e[:, :2] - want) <= 1e-10 * mag)
