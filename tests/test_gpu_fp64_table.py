"""The FP64 table of erfc(alpha r)/r (grx_table.cu), one pair at a time, against 30 digits: a bead and an
atom of charge 1 on an axis, at distances with an exact square, so that an energy is the table's value
and one rounding of the product with the prefactor. The table states an rms error of 1.0e-16; a rounding
is 0.64e-16 rms at worst (half of 2^-53 to 2^-52, evenly): 1.2e-16 together, 1.5e-16 asked for, and
5e-16 for the largest of 2,000."""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [0.2, 0.265])
def test_error_of_one_evaluation(grx_lib, alpha):
    mp = pytest.importorskip("mpmath")
    s = synth.silica_co2(alpha=alpha)
    s["molsize"] = [1, 3]
    synth._set_atoms(s, np.zeros((1, 3)), s["type"][:1], np.ones(1), [np.zeros((0, 3))])
    s["epsilon"] = np.zeros_like(s["epsilon"])
    box = grx_lib.Box(s, capacity=[1, 64])
    n = 2000
    k = np.random.default_rng(3).integers(int(0.52 * 2 ** 22), int(11.99 * 2 ** 22), n)
    x = k / 2.0 ** 22  # 26 bits: x * x is exact
    pos = np.zeros((n, 3))
    pos[:, 0] = x
    e, _ = box.trial_energies(pos, np.ones(n), np.full(n, 3), 10 ** 6, n, 1, 1, prec=grx_lib.GRX_FP64)
    with mp.workdps(30):
        a, pre = mp.mpf(float(s["alpha"])), mp.mpf(float(s["prefactor"]))
        rel = np.array([float(mp.mpf(float(v)) / (pre * mp.erfc(a * mp.mpf(float(r))) / mp.mpf(float(r))) - 1)
                        for v, r in zip(e[:, 1], x)])
    assert np.sqrt(np.mean(rel ** 2)) <= 1.5e-16
    assert np.abs(rel).max() <= 5e-16
