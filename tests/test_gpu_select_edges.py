"""Widom insertions at the edges of a Rosenbluth step's lane layout (1, 31, 32, 33, 64 trials) and of
a pass's nearest-atoms-first split (all trials overlapping, none, chains of one and three beads,
more beads than the split takes), against the FP64 oracle: identical selections and counts of
trials without overlap, energies of the chosen trials to the FP64 bar 1e-12 max(|E|, 1), weights to
1e-10 (an energy of 1e4 kT at that bar). The real Coulomb parts sum 400 pairs per bead of either
sign, up to 138935 x 0.7 x 2.05 / 1.6 = 1e5 each: their roundings alone reach 400 x 1e5 x 1.1e-16
on either side, so 1e-8 is added to their bar."""
import numpy as np
import pytest

from graspa_gb300 import synth
from tests.test_gpu_parity import oracle_widom

pytestmark = pytest.mark.gpu


def _check(grx_lib, s, ntrials, norient, n):
    ref, _ = oracle_widom(s, 1, n, ntrials=ntrials, norient=norient)
    box = grx_lib.Box(s, capacity=[s["comp_start"][1], 3 * 64])
    box.ewald_total()
    got = box.widom(grx_lib.widom_desc(s, 1, ntrials, norient), 0, n, prec=grx_lib.GRX_FP64)
    for k in ("sel_first", "sel_orient", "n_ok_first", "n_ok_orient", "success"):
        assert np.array_equal(got[k], [getattr(r, k) for r in ref]), k
    for k in ("e_first", "e_chain"):
        want = np.array([list(getattr(r, k)) for r in ref])
        bar = 1e-12 * np.maximum(np.abs(want), 1.0) + np.array([0.0, 1e-8, 0.0, 1e-8])
        assert np.all(np.abs(got[k] - want) <= bar), k
    w = np.array([r.rosenbluth for r in ref])
    assert np.all(np.abs(got["rosenbluth"] - w) <= 1e-10 * np.abs(w))
    return got


@pytest.mark.parametrize("norient", [1, 10])
@pytest.mark.parametrize("ntrials", [1, 31, 32, 33, 64])
def test_trial_counts(grx_lib, ntrials, norient):
    _check(grx_lib, synth.silica_co2(n_co2=4), ntrials, norient, 24)


def test_more_beads_than_the_near_split(grx_lib):
    got = _check(grx_lib, synth.silica_co2(n_co2=4), 20, 64, 16)  # 128 beads
    assert np.any(got["success"])


@pytest.mark.parametrize("overlap", [1e-3, 1e300])
def test_all_or_no_trials_overlap(grx_lib, overlap):
    s = synth.silica_co2()
    s["overlap_criteria"] = overlap
    got = _check(grx_lib, s, 12, 7, 24)
    if overlap < 1:
        assert np.any(got["n_ok_first"] < 12)
