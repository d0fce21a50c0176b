"""The FP64 pair evaluation (FP32 screening and image choice, tabulated erfc) against the FP64
oracle where it changes path: distances from 0.05 A (library functions below 0.5 A) to past the
cutoff, fractions next to half a cell, unwrapped and far coordinates (images by rounded FP64
fractions), cells narrower than twice the cutoff, lambda-scaled beads, the tile path.

Bar per trial and part: 1e-12 times the sum of the pair energies' magnitudes, for trials whose
nearest atom is at least 0.25 A away (a displacement carries about 1.5e-14 A of rounding, on
either side, which r^-12 amplifies by 12 / r; nearer trials compare their flags). Far beads
(|x| ~ 4000 A) carry 1e-12 A: 1e-9.
"""
import numpy as np
import pytest

from graspa_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _system(which):
    if which == "silica":
        return synth.silica_co2(n_co2=6)
    if which == "narrow":  # 20.1 x 19.7 x 26.3 A against a 12 A cutoff: the tile path, ties inside the cutoff
        return synth.silica_co2(cells=(1, 1, 2), kmax=(5, 5, 6), n_co2=3)
    if which == "water":
        return synth.tip4p_hex_system(n_water=6)
    s = synth.ch4_xe_system(5, n_ch4=3, n_xe=3)
    return s


def _beads(s, rng):
    """Beads at chosen distances of framework atoms, next to half-cell fractions of them, and at random."""
    cell = np.array(s["cell"]).reshape(3, 3)
    fw = s["pos"][:s["comp_start"][1]]
    pick = lambda n: fw[rng.integers(0, len(fw), n)]  # noqa: E731
    dirs = lambda n: (lambda v: v / np.linalg.norm(v, axis=1, keepdims=True))(rng.normal(size=(n, 3)))  # noqa: E731
    r = np.array([0.05, 0.09, 0.11, 0.3, 0.4999, 0.5001, 0.9, 1.7, 2.4, 3.3, 6.0, 10.0, s["cutoff_vdw"] - 1e-7, s["cutoff_vdw"] + 1e-7])
    near = pick(len(r)) + r[:, None] * dirs(len(r))
    half = pick(12) + (0.5 * np.eye(3)[rng.integers(0, 3, 12)] + rng.normal(scale=2e-6, size=(12, 3))) @ cell
    return np.concatenate([near, half, rng.uniform(0, 1, (6, 3)) @ cell])


def _magnitudes(s, pos, q, ty, scale):
    """Nearest distance and sums of |pair energy| (host vdw, host real, guest vdw, guest real) of each bead."""
    cell, nt = np.array(s["cell"]).reshape(3, 3), s["ntypes"]
    f = (s["pos"][None, :, :] - pos[:, None, :]) @ np.linalg.inv(cell)
    r2 = (((f - np.round(f)) @ cell) ** 2).sum(2)
    row = (s["type"][None, :], ty[:, None])
    eps, sig, sh = (np.asarray(s[k]).reshape(nt, nt)[row] for k in ("epsilon", "sigma", "shift"))
    r2f = np.maximum(r2, 1e-20)
    t3 = (r2f / sig ** 2) ** 3 + 0.5 * (1 - scale) ** 2
    lj = np.where(r2 < s["cutoff_vdw"] ** 2, scale * (4 * eps * (1 / t3 ** 2 + 1 / t3) + np.abs(sh)), 0.0)
    co = np.where((r2 < s["cutoff_coul"] ** 2) & (not s["no_charges"]),
                  s["prefactor"] * np.abs(s["charge"][None, :] * q[:, None]) * scale / np.sqrt(r2f), 0.0)
    h = s["comp_start"][1]
    return np.sqrt(r2.min(1)), np.stack([lj[:, :h].sum(1), co[:, :h].sum(1), lj[:, h:].sum(1), co[:, h:].sum(1)], 1)


@pytest.mark.parametrize("scale", [1.0, 0.6])
@pytest.mark.parametrize("which", ["silica", "narrow", "water", "ch4_xe"])
def test_fp64_pairs(grx_lib, which, scale):
    s = _system(which)
    comp = 1
    box = grx_lib.Box(s, capacity=[s["comp_start"][1]] + [64] * (len(s["molsize"]) - 1))
    S = O.OracleSystem(s)
    rng = np.random.default_rng(21)
    pos = _beads(s, rng)
    n = len(pos)
    cell = np.array(s["cell"]).reshape(3, 3)
    tm = s["templates"][comp]
    q, ty = np.full(n, tm["charge"][-1]), np.full(n, tm["type"][-1])
    nearest, mag = _magnitudes(s, pos, q, ty, scale)
    sc = np.full(n, scale)
    for lattice, bar in (((0, 0, 0), 1e-12), ((1, -1, 0), 1e-12), ((-3, 2, 1), 1e-12), ((100, 0, -150), 1e-9)):
        p = pos + np.array(lattice) @ cell
        e, f = box.trial_energies(p, q, ty, 10 ** 6, n, 1, comp, prec=grx_lib.GRX_FP64, scale=sc, scale_coul=sc)
        r, rf = S.trial_energies(p, sc, q, sc, ty, 10 ** 6, n, 1, comp)
        assert np.array_equal(f, rf)
        keep = nearest >= 0.25
        assert keep.sum() >= n // 2
        assert np.all(np.abs(e - r)[keep] <= bar * (1.0 + mag)[keep]), (lattice, np.abs(e - r).max())


@pytest.mark.parametrize("alpha", [0.05, 0.265, 0.9])
def test_fp64_tables_over_alpha(grx_lib, alpha):
    """alpha 0.9: the Gaussian tail past alpha^2 s = 20 takes the library erfc."""
    s = synth.silica_co2(alpha=alpha, n_co2=4)
    box = grx_lib.Box(s, capacity=[s["comp_start"][1], 64])
    rng = np.random.default_rng(5)
    pos = rng.uniform(0, 1, (64, 3)) @ np.array(s["cell"]).reshape(3, 3)
    q, ty, one = np.full(64, -0.35), np.full(64, 3), np.ones(64)
    e, _ = box.trial_energies(pos, q, ty, 10 ** 6, 64, 1, 1, prec=grx_lib.GRX_FP64)
    r, _ = O.OracleSystem(s).trial_energies(pos, one, q, one, ty, 10 ** 6, 64, 1, 1)
    nearest, mag = _magnitudes(s, pos, q, ty, 1.0)
    keep = nearest >= 0.25
    assert np.all(np.abs(e - r)[keep] <= 1e-12 * (1.0 + mag)[keep])
