"""Voxel lists of cells narrower than twice the list radius (images by rounded fractions): the same
trial energies and overlap flags as the tile path, for an orthorhombic cell narrower than the
cutoff's diameter, a skewed one, beads next to half-cell ties and outside the home cell.

Bar: the same pairs in another order, 1e-12 of a bound of the sum of their magnitudes."""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


def _system(which):
    if which == "orthorhombic":
        return synth.silica_co2(cells=(1, 1, 2), kmax=(5, 5, 6), n_co2=3)
    if which == "hexagonal":
        return synth.tip4p_hex_system(n_water=4)
    return synth.adsorbate_system("CO2", 11, n_atoms=1500, n_guest=3)  # 25 A wide, strongly skewed


@pytest.mark.parametrize("prec", ["mixed", "fp64", "fp32"])
@pytest.mark.parametrize("which", ["orthorhombic", "hexagonal", "skewed"])
def test_narrow_lists_match_tiles(grx_lib, which, prec):
    s = _system(which)
    cap = [s["comp_start"][1], 64]
    vox, tile = grx_lib.Box(s, capacity=cap), grx_lib.Box(s, capacity=cap)
    tile.set_voxel_lists(0)
    assert vox.voxel_lists()[0] and not tile.voxel_lists()[0]
    rng = np.random.default_rng(8)
    cell = np.array(s["cell"]).reshape(3, 3)
    fw = s["pos"][:cap[0]]
    n = 120
    pos = rng.uniform(-1, 2, (n, 3)) @ cell
    pos[:30] = fw[rng.integers(0, cap[0], 30)] + (0.5 * np.eye(3)[rng.integers(0, 3, 30)] +
                                                  rng.normal(scale=1e-5, size=(30, 3))) @ cell
    tm = s["templates"][1]
    q, ty = np.full(n, tm["charge"][-1]), np.full(n, tm["type"][-1])
    p = grx_lib.PRECISIONS[prec]
    (e, f), (g, h) = (b.trial_energies(pos, q, ty, 10 ** 6, n, 1, 1, prec=p) for b in (vox, tile))
    assert np.array_equal(f, h)
    mag = s["prefactor"] * abs(tm["charge"][-1]) * np.abs(s["charge"]).max() * 1000
    ok = np.isfinite(g)  # beads on top of a replicated atom: not finite on either path
    assert np.array_equal(ok, np.isfinite(e)) and ok.sum() > 400
    assert np.all(np.abs(e - g)[ok] <= 1e-12 * (mag + np.abs(g))[ok])
