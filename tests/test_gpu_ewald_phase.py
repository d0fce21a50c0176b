"""Phases of the mixed Fourier delta: guests 50 cells from home, whose fractions are large. 40 mixed
GCMC translations of far CO2; the adsorbate structure factor they commit against the one recomputed
in FP64 from the final positions.

Bar: with the whole cells taken off, an entry e^{2 pi i k f} rounds its phase by at most
2 pi (k / 2) 3 x 2^-49 (split and product), 1.5e-13 at k = 9, and a move has 3 atoms of charges 1.4 in
all, old and new, with three such factors: 1.3e-12 at most. Ten moves' worth, 1.3e-11, for 40 whose
errors have either sign. (FP64 fractions of 50 carry 1e-14 on either side.) With the cells left in, the
bound is a hundred times that."""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(0, 0, 0), (50, -50, 50)])
@pytest.mark.parametrize("kmax", [(9, 9, 6), (2, 2, 20)])  # by columns, and with (kx, ky) row products
def test_committed_phases(grx_lib, kmax, cells):
    s = synth.silica_co2(kmax=kmax, n_co2=6)
    nfw = s["comp_start"][1]
    s["pos"] = s["pos"].copy()
    s["pos"][nfw:] += np.array(cells) @ np.array(s["cell"]).reshape(3, 3)
    box = grx_lib.Box(s, capacity=[nfw, 3 * 64])
    box.total_energy()
    d = grx_lib.gcmc_desc(1, p_translation=1.0, p_rotation=1.0, p_reinsertion=1.0, p_swap=1.0, pressure_pa=1e6, seed=9)
    st = grx_lib.gcmc_run([box], [d], 0, 40, grx_lib.GRX_MIXED)[0]
    assert st.accepted[0] >= 5
    got = box.structure_factors()[1]
    box.total_energy()
    scale = max(kmax) / 9
    assert np.max(np.abs(got - box.structure_factors()[1])) <= 1.3e-11 * scale
