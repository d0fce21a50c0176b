"""The mixed pair path where its list walk and Coulomb table change branch: voxel lists against the
tile path (whole chunks of certain entries, the screened rest, an excluded framework molecule,
which sends every entry through the screen) and against the FP64 form, over distances across the
table's pieces and below it.

Bars: lists against tiles the same pairs in another order, 1e-12 of the sum of the magnitudes; mixed
against FP64 the mixed bar beta |dE| <= 1e-6 on trials without overlap.
"""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


def _system(which):
    if which == "silica":
        return synth.silica_co2(n_co2=5)
    return synth.adsorbate_system("CO2", 9, n_atoms=1500, n_guest=3)


@pytest.mark.parametrize("exclude_host", [False, True])
@pytest.mark.parametrize("which", ["silica", "triclinic"])
@pytest.mark.parametrize("ntrials", [1, 7, 64])
def test_voxel_walk(grx_lib, which, exclude_host, ntrials):
    s = _system(which)
    cap = [s["comp_start"][1], 64]
    rng = np.random.default_rng(31 + ntrials)
    cell = np.array(s["cell"]).reshape(3, 3)
    if exclude_host:  # the framework as single-atom molecules: one of them is left out
        s = dict(s)
        s["molsize"] = [1, 3]
        s["molid"] = np.concatenate([np.arange(cap[0]), s["molid"][cap[0]:]])
    vox, tile = grx_lib.Box(s, capacity=cap), grx_lib.Box(s, capacity=cap)
    tile.set_voxel_lists(0)
    assert vox.voxel_lists()[0] and not tile.voxel_lists()[0]
    near = s["pos"][rng.integers(0, cap[0], ntrials)]
    v = rng.normal(size=(ntrials, 3))
    r = np.exp(rng.uniform(np.log(0.4), np.log(6.0), (ntrials, 1)))
    pos = near + r * v / np.linalg.norm(v, axis=1, keepdims=True)
    pos[ntrials // 2:] = rng.uniform(-1, 2, (ntrials - ntrials // 2, 3)) @ cell
    q, ty = np.full(ntrials, -0.35), np.full(ntrials, s["templates"][1]["type"][-1])
    ex = dict(excl_comp=0, excl_molid=int(rng.integers(0, cap[0]))) if exclude_host else {}
    out = {}
    for name, b in (("vox", vox), ("tile", tile)):
        for prec in ("mixed", "fp64"):
            out[name, prec] = b.trial_energies(pos, q, ty, 10 ** 6, ntrials, 1, 1, prec=grx_lib.PRECISIONS[prec], **ex)
    mag = s["prefactor"] * 0.35 * np.abs(s["charge"]).max() * 800 / 0.4
    for prec in ("mixed", "fp64"):
        (e, f), (g, h) = out["vox", prec], out["tile", prec]
        assert np.array_equal(f, h)
        assert np.all(np.abs(e - g) <= 1e-12 * (mag + np.abs(g)))
    (e, f), (g, h) = out["vox", "mixed"], out["vox", "fp64"]
    assert np.array_equal(f, h)
    ok = f == 0
    assert np.all(grx_lib.beta_from_temperature(300.0) * np.abs(e - g)[ok] <= 1e-6)
