"""Boxes without a cutoff (infinite squared cutoffs): every pair counts at its rounded image. Box
creation sizes its tables by the cell then; FP64 and mixed energies against a sum over all pairs.

Bars, with M the sum of the magnitudes of a trial's pair terms (atoms at least 2 A away: a term changes
by at most 6 of itself per A): 1e-12 M in FP64, 1e-6 M + 1e-6 kT in the mixed form."""
import numpy as np
import pytest
from scipy.special import erfc

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["silica", "skewed"])
def test_infinite_cutoffs(grx_lib, which):
    s = synth.silica_co2(n_co2=3) if which == "silica" else synth.adsorbate_system("CO2", 11, n_atoms=1500, n_guest=3)
    s["cutoff_vdw"] = s["cutoff_coul"] = np.inf
    h = s["comp_start"][1]
    box = grx_lib.Box(s, capacity=[h, 64])
    rng = np.random.default_rng(6)
    cell, nt = np.array(s["cell"]).reshape(3, 3), s["ntypes"]
    p = rng.uniform(0, 1, (200, 3)) @ cell
    f = (s["pos"][None] - p[:, None]) @ np.linalg.inv(cell)
    r = np.linalg.norm((f - np.round(f)) @ cell, axis=2)
    p, r = p[r.min(1) > 2.0], r[r.min(1) > 2.0]
    n = len(p)
    assert n >= 10
    tm = s["templates"][1]
    q, ty = np.full(n, tm["charge"][-1]), np.full(n, tm["type"][-1])
    row = (s["type"][None, :], ty[:, None])
    eps, sig, sh = (np.asarray(s[k]).reshape(nt, nt)[row] for k in ("epsilon", "sigma", "shift"))
    t = (sig / r) ** 6
    lj = 4 * eps * (t * t - t) - sh
    co = s["prefactor"] * s["charge"][None] * q[:, None] * erfc(s["alpha"] * r) / r
    parts = (lj[:, :h], co[:, :h], lj[:, h:], co[:, h:])
    want = np.stack([x.sum(1) for x in parts], 1)
    mag = np.stack([np.abs(x).sum(1) for x in parts], 1) + np.stack([4 * eps[:, k].max(1) for k in
                                                                     (slice(0, h), slice(0, h), slice(h, None), slice(h, None))], 1)
    for prec, bar in ((grx_lib.GRX_FP64, 1e-12 * mag),
                      (grx_lib.GRX_MIXED, 1e-6 * mag + 1e-6 / grx_lib.beta_from_temperature(300.0))):
        e, flags = box.trial_energies(p, q, ty, 10 ** 6, n, 1, 1, prec=prec)
        assert not flags.any()
        assert np.all(np.abs(e - want) <= bar), prec
